// Dense block-FP8 GEMM for few rows, bound by reading the weights:
//     out[m, n] = sum_kb (X[m, kb] . W[n, kb]) * xs[m, kb] * Bs[n / 128, kb]
// Operands are swapped as in gemm_stream.cuh: a CTA owns 256 weight rows (two UMMA tiles of 128), NT = 16 / 32 / 64 tokens
// are the UMMA N dimension. K is split over a thread-block cluster of up to 8 CTAs so that about every SM streams
// weights, and the partial sums are exchanged through distributed shared memory: no fp32 partials in memory and no
// reduction launch. The first weight tiles are on their way into L2 before the kernels
// ahead in the stream have finished.
//   QUANT = true: X is the 16-bit input of a linear layer of a few rows (NT = 16); every CTA quantises its K range once,
//       up front (same bytes and scales as the stand-alone quantiser), and keeps it in shared memory for all of its
//       weight tiles: quantiser, GEMM and sum in ONE launch.
//   QUANT = false: X is FP8 with its scales, loaded by TMA next to the weights.
//   warps 0-7  (quantise,) promote: lane = weight row, columns = tokens
//   warp  8    TMA producer
//   warp  9    MMA issuer
#pragma once

#include "gemm_stream.cuh"

namespace b200 {

struct LinearStreamParams {
  const void* x;    // QUANT: [M, K] 16-bit, row-major
  const float* As;  // otherwise: scales As[m * as_sm + kb * as_sk]
  int64_t as_sm, as_sk;
  const float* Bs;  // [ceil(N/128)][num_kb]
  void* out;        // OutT [M, N]
  int M, N, K, num_kb, kb_per_rank;
  int n_tiles, t_tiles, stages;
  const uint8_t* w;  // the weights [N, K]
  int own_sums;  // a cluster's sums have a place outside the ring
  float eps;
  int* status;
};

template <int NT, bool QUANT>
struct LinearStreamCfg {
  static constexpr int kThreads = 320, kMinCtas = NT <= 32 ? 2 : 1;
  static constexpr int kStageW = 256 * kBK, kStageX = QUANT ? 0 : NT * kBK, kStage = kStageW + kStageX;
  // per K block of the CTA: (tokens,) their scales, two weight scales
  static constexpr int kKbBytes = (QUANT ? NT * kBK : 0) + NT * 4 + 8;
  static constexpr int kAccBufs = NT == 64 ? 2 : 4, kTmemCols = kAccBufs * 2 * NT;
  static constexpr int kFixed = 1024 + 512;
  static constexpr int kSmemLimit = 232448, kHalfSm = 115 * 1024;  // two CTAs per SM: 228 KB less 1 KB each
  static constexpr int kMaxStages = 6;
  static size_t smem_for(int stages, int kb) { return (size_t)stages * kStage + (size_t)kb * kKbBytes + kFixed; }
};

// T: type of the output (and of x, QUANT)
template <int NT, bool QUANT, typename T>
__global__ void __launch_bounds__(LinearStreamCfg<NT, QUANT>::kThreads, LinearStreamCfg<NT, QUANT>::kMinCtas)
linear_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                     const LinearStreamParams p) {
  using Cfg = LinearStreamCfg<NT, QUANT>;
  constexpr int NB = Cfg::kAccBufs;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const int S = p.stages, cap = p.kb_per_rank;
  const uint32_t sW = smem_base, sX = smem_base + S * Cfg::kStageW;
  uint8_t* x_ptr = smem_al + (size_t)S * Cfg::kStageW;  // [kb or stage][NT x 128 bytes, 128-byte swizzle]
  uint64_t* bars = reinterpret_cast<uint64_t*>(x_ptr + (size_t)(QUANT ? cap : S) * NT * kBK);
  float* table = reinterpret_cast<float*>(bars + 32);                   // [kb][NT] row scales
  float* bs_tab = table + cap * NT;                                     // [2][kb] weight-block scales
  const uint32_t bar0 = ptx::smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (8 + s); };
  auto tfull_bar = [&](int b) { return bar0 + 8u * (16 + b); };
  auto tempty_bar = [&](int b) { return bar0 + 8u * (16 + NB + b); };
  const uint32_t x_bar = bar0 + 8u * (16 + 2 * NB);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 17 + 2 * NB);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 18 + 2 * NB);

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
    ptx::mbar_init(x_bar, 8);
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), Cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  if (warp == kProducerWarp && lane == 0) {
    ptx::prefetch_tensormap(&tmap_w);
    if (!QUANT) ptx::prefetch_tensormap(&tmap_x);
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // "I have started", waited for before another CTA's shared memory is written at the very end
  if (csize > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  // The next kernels may start: at once behind the one-launch kernel (four projections of 1 row, rank of eight, 19.9 us in a
  // graph, signalled at the end of the K loop 21.5), else there, as in gemm_skinny.cuh. After the TMEM allocation in any
  // case: a dependent grid's CTA that got its columns first, and then waits for this grid, would otherwise hold them for ever.
  if (QUANT) grid_launch_dependents();

  const int item0 = blockIdx.x / csize, step = gridDim.x / csize;
  const int kb0 = (int)rank * p.kb_per_rank, kb1 = min(p.num_kb, kb0 + p.kb_per_rank);
  const int nkb = max(kb1 - kb0, 0);
  const int row_blocks = (p.N + 127) / 128;
  const int items = p.n_tiles * p.t_tiles;  // the token tiles of one weight tile side by side: they share it in L2

  float acc[NT];
  bool sum_ok = false;
  const int half = warp >> 2, r = threadIdx.x & 127;
  auto store = [&](int item) {
    const int nt = item / p.t_tiles, m0 = (item - nt * p.t_tiles) * NT;
    const int n = nt * 256 + half * 128 + r;
    if (n < p.N) {
      T* out = static_cast<T*>(p.out) + n;
#pragma unroll
      for (int t = 0; t < NT; ++t)  // 32 lanes -> 32 consecutive n
        if (m0 + t < p.M) out[(int64_t)(m0 + t) * p.N] = from_f32<T>(acc[t]);
    }
  };

  if (warp == kProducerWarp) {
    if (ptx::elect_one()) {
      int s = 0;
      uint32_t phase = 1;
      bool ok = true;
      grid_dependency_wait();
      for (int item = item0; item < items && ok; item += step) {
        const int nt = item / p.t_tiles, m0 = (item - nt * p.t_tiles) * NT;
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = ptx::mbar_wait(empty_bar(s), phase, abort_flag);
          if (!ok) break;
          ptx::mbar_expect_tx(full_bar(s), Cfg::kStage);
          ptx::tma_load_2d(sW + s * Cfg::kStageW, &tmap_w, kb * kBK, nt * 256, full_bar(s));
          ptx::tma_load_2d(sW + s * Cfg::kStageW + 128 * kBK, &tmap_w, kb * kBK, nt * 256 + 128, full_bar(s));
          if (!QUANT) ptx::tma_load_2d(sX + s * Cfg::kStageX, &tmap_x, kb * kBK, m0, full_bar(s));
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
      bool ok = !QUANT || ptx::mbar_wait(x_bar, 0, abort_flag);
      for (int item = item0; item < items && ok; item += step) {
        for (int j = 0; j < nkb; ++j, ++it) {
          const int b = it % NB;
          ok = ptx::mbar_wait(tempty_bar(b), ((it / NB) & 1) ^ 1, abort_flag) &&
               ptx::mbar_wait(full_bar(s), phase, abort_flag);
          if (!ok) break;
          ptx::tc_fence_after();
          const uint64_t dw = ptx::smem_desc_sw128(sW + s * Cfg::kStageW);
          const uint64_t dx = ptx::smem_desc_sw128(sX + (QUANT ? j : s) * NT * kBK);
          const uint32_t d = tmem_base + b * 2 * NT;
#pragma unroll
          for (int h = 0; h < 2; ++h)
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
  } else {
    // Every operand and the output buffer belong to the kernels before this one, which may still run. The weight stream
    // starts all the same, as a prefetch into L2, a row for each thread.
    const int n_first = item0 / p.t_tiles * 256 + threadIdx.x;
    if (n_first < p.N) prefetch_weight_row(p.w + (int64_t)n_first * p.K + kb0 * kBK, min(kPrefetchKb, nkb));
    grid_dependency_wait();
    if constexpr (QUANT) {
      // 8 lanes share the 128-group of one row, 32 groups in flight per round: (K block, row) = group index
      const int chunk = threadIdx.x & 7;
      const int groups = nkb * p.M;
      // the loads of four rounds are in flight before the first is used: an L2 round trip is as long as a round
      constexpr int R = 4;
      for (int g0 = threadIdx.x >> 3; g0 - (threadIdx.x >> 3) < groups; g0 += 32 * R) {
        uint4 raw[R][2];
        int kb[R], row[R];
#pragma unroll
        for (int u = 0; u < R; ++u) {
          const int g = g0 + 32 * u;
          kb[u] = g < groups ? g / p.M : -1;
          row[u] = g - kb[u] * p.M;
          const bool in = kb[u] >= 0 && (kb0 + kb[u]) * 128 + chunk * 16 < p.K;  // K is a multiple of 16
          const T* src = static_cast<const T*>(p.x) + (int64_t)row[u] * p.K + (int64_t)(kb0 + kb[u]) * 128 + chunk * 16;
          raw[u][0] = in ? ld_nc_16(src) : make_uint4(0, 0, 0, 0);
          raw[u][1] = in ? ld_nc_16(src + 8) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < R; ++u) {
          if (g0 - (threadIdx.x >> 3) + 32 * u >= groups) break;  // the same for every thread
          uint4 q;
          const float sc = quant_chunk<T>(raw[u], p.eps, q);
          if (kb[u] >= 0) {
            *reinterpret_cast<uint4*>(x_ptr + (size_t)kb[u] * NT * kBK + (row[u] >> 3) * 1024 + (row[u] & 7) * 128 +
                                      ((chunk ^ (row[u] & 7)) << 4)) = q;
            if (chunk == 0) table[kb[u] * NT + row[u]] = sc;
          }
        }
      }
    }
    if (QUANT) {
      ptx::fence_proxy_async_smem();  // generic-proxy writes -> the tensor core's reads
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(x_bar);
    }
    const uint32_t lane_base = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + half * NT;
    uint32_t it = 0;
    bool ok = true;
    for (int item = item0; item < items && ok; item += step) {
      const int nt = item / p.t_tiles, m0 = (item - nt * p.t_tiles) * NT;
      named_bar_sync(1, 256);  // every warp is done with the last item's tables
      for (int i = threadIdx.x; i < 2 * nkb; i += 256) {
        const int h = i >= nkb, kb = i - h * nkb;
        bs_tab[h * cap + kb] = __ldg(p.Bs + (int64_t)min(nt * 2 + h, row_blocks - 1) * p.num_kb + kb0 + kb);
      }
      if (!QUANT) {
#pragma unroll 4
        for (int i = threadIdx.x; i < nkb * NT; i += 256) {
          const int j = i / NT, m = min(m0 + i % NT, p.M - 1);
          table[i] = __ldg(p.As + (int64_t)m * p.as_sm + (int64_t)(kb0 + j) * p.as_sk);
        }
      }
      named_bar_sync(1, 256);
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[t] = 0.f;
      for (int j = 0; j < nkb && ok; ++j, ++it) {
        const int b = it % NB;
        ok = ptx::mbar_wait(tfull_bar(b), (it / NB) & 1, abort_flag);
        if (!ok) break;
        ptx::tc_fence_after();
        const float bs = bs_tab[half * cap + j];
        const float4* sc = reinterpret_cast<const float4*>(table + j * NT);
        constexpr int CH = NT < 32 ? NT : 32;
        // columns past M hold whatever the rows past M of the x tile gave; they are never stored
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
      if (csize > 1) break;  // one item per cluster: finished below
      if (ok) store(item);
    }
    if (!QUANT) grid_launch_dependents();
    if (csize > 1) sum_ok = !named_bar_any(1, 256, !ok);
  }

  if (csize > 1) {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    // every rank adds up its share of the tokens (token t belongs to rank t / per): [rank][token][row], behind the tables, or
    // in the ring, which is idle once every rank is here
    if (!p.own_sums) ptx::cluster_sync();
    const uint32_t sums_off = p.own_sums ? (uint32_t)(reinterpret_cast<uint8_t*>(bs_tab + 2 * cap) - smem_al + 15) & ~15u : 0u;
    const int nt = item0 / p.t_tiles, m0 = (item0 - nt * p.t_tiles) * NT;
    const int rows = min(NT, p.M - m0), per = (rows + (int)csize - 1) / (int)csize, n = half * 128 + r;
    if (warp < 8) {
      int owner = 0, j = 0;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        if (t < rows) ptx::st_cluster_f32(ptx::mapa(smem_base + sums_off, owner) + (((int)rank * per + j) * 256 + n) * 4, acc[t]);
        if (++j == per) j = 0, ++owner;
      }
    }
    __syncwarp();
    ptx::cluster_sync();
    if (warp < 8 && sum_ok && nt * 256 + n < p.N) {
      const float* src = reinterpret_cast<const float*>(smem_al + sums_off) + n;
      T* out = static_cast<T*>(p.out) + nt * 256 + n;
      const int t0 = (int)rank * per, n_mine = min(per, rows - t0);
      constexpr int U = NT == 16 ? 2 : 8;  // rows in flight
      for (int j = 0; j < n_mine; j += U) {
        float sum[U];
#pragma unroll
        for (int u = 0; u < U; ++u) sum[u] = 0.f;
        for (int c = 0; c < (int)csize; ++c)  // rank order: the same sum on every run
#pragma unroll
          for (int u = 0; u < U; ++u) sum[u] += src[(c * per + min(j + u, n_mine - 1)) * 256];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (j + u < n_mine) out[(int64_t)(m0 + t0 + j + u) * p.N] = from_f32<T>(sum[u]);
      }
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

inline int64_t linear_sum_bytes(int64_t csize, int64_t rows) { return csize * cdiv(rows, csize) * 1024 + 16; }

// Cluster size and ring depth; false when nothing fits.
template <int NT, bool QUANT>
inline bool plan_linear_stream(int64_t M, int64_t N, int64_t K, int sms, int& csize, int& kb_per_rank, int& stages, int& own_sums) {
  using Cfg = LinearStreamCfg<NT, QUANT>;
  const int64_t items = cdiv(N, 256) * cdiv(M, NT), num_kb = cdiv(K, kBK), rows = M < NT ? M : NT;
  // as many ranks per item as bring items x ranks up to the SM count, two K blocks each at least; where a rank could not
  // hold its K range, or the ring not the other ranks' sums, the nearest cluster size that fits
  int64_t want = sms / items;
  // Clusters of up to 8 as long as they all run at once, at one CTA per SM: the SM groups of this part hold 15 of them
  // (cudaOccupancyMaxActiveClusters), which depends on the SMs that a part has, so one is left spare. Clusters of 4 (33 fit)
  // beyond. With weights from HBM, 8 against 4: 13 tiles, 1 x 3328 x 4096 6.1 and 7.3 us, 61 x 3328 x 14336 18.7 and 22.5;
  // 14 tiles 6.2 and 7.3, 19.1 and 22.8; 15 tiles 6.4 and 7.4, 19.9 and 22.6; 16 tiles 7.7 and 7.7, 32.3 and 22.5.
  if (want > 4) want = items <= 14 ? 8 : 4;
  if (want > num_kb / 2) want = num_kb / 2;
  if (want < 1) want = 1;
  for (int i = 0; i < 16; ++i) {
    const int64_t c = i % 2 ? want + i / 2 : want - i / 2;
    if (c < 1 || c > 8) continue;
    kb_per_rank = (int)cdiv(num_kb, c);
    csize = (int)cdiv(num_kb, kb_per_rank);  // no rank without work
    // two CTAs on an SM if a ring of three stages fits: the next projection's CTAs then fill theirs while this one drains
    const int64_t tail = (int64_t)kb_per_rank * Cfg::kKbBytes + Cfg::kFixed;
    int64_t s = Cfg::kMinCtas == 2 ? (Cfg::kHalfSm - tail) / Cfg::kStage : 0;
    if (s < 3) s = (Cfg::kSmemLimit - tail) / Cfg::kStage;
    stages = (int)(s < Cfg::kMaxStages ? s : Cfg::kMaxStages);
    // the ranks' sums (1 KB per row) get a place of their own where that costs the ring no stage it needs (64 KB of 64-token sums took two of
    // five: 61 rows, four projections of a rank of four 76 -> 79.5 us), else they land in the ring, one more barrier later
    const int64_t sums = linear_sum_bytes(csize, rows);
    const bool half = Cfg::kMinCtas == 2 && (int64_t)stages * Cfg::kStage + tail <= Cfg::kHalfSm;
    const int64_t left = ((half ? Cfg::kHalfSm : Cfg::kSmemLimit) - tail - sums) / Cfg::kStage;
    own_sums = csize > 1 && (left >= 5 || left >= (stages < Cfg::kMaxStages ? stages : Cfg::kMaxStages));
    if (own_sums) stages = (int)(left < Cfg::kMaxStages ? left : Cfg::kMaxStages);
    if (own_sums || (stages >= 2 && (csize == 1 || sums <= (int64_t)stages * Cfg::kStage))) return true;
  }
  return false;
}

// X: FP8 rows (QUANT: unused, p.x holds the 16-bit rows)
template <int NT, bool QUANT, typename T>
inline int launch_linear_stream(const void* W, const void* X, LinearStreamParams p, cudaStream_t st) {
  using Cfg = LinearStreamCfg<NT, QUANT>;
  const int sms = sm_count();
  int csize;
  p.num_kb = (int)cdiv(p.K, kBK);
  p.n_tiles = (int)cdiv(p.N, 256);
  p.t_tiles = (int)cdiv(p.M, NT);
  if (!plan_linear_stream<NT, QUANT>(p.M, p.N, p.K, sms, csize, p.kb_per_rank, p.stages, p.own_sums)) {
    set_error_detail("linear_stream: K=%d does not fit shared memory", p.K);
    return B200_E_UNSUPPORTED;
  }
  p.status = device_status_word();
  if (!p.status) {
    set_error_detail("cannot resolve the device status word");
    return B200_E_LAUNCH;
  }
  p.w = static_cast<const uint8_t*>(W);
  CUtensorMap tw, tx;
  int rc = make_tmap_u8(&tw, W, (uint64_t)p.N, (uint64_t)p.K, 128, "W");
  if (rc) return rc;
  tx = tw;
  if (!QUANT && (rc = make_tmap_u8(&tx, X, (uint64_t)p.M, (uint64_t)p.K, (uint32_t)NT, "X"))) return rc;
  auto k = linear_stream_kernel<NT, QUANT, T>;
  if (int rc_smem = allow_smem(k, Cfg::kSmemLimit, "linear_stream_kernel")) return rc_smem;
  const int64_t items = (int64_t)p.n_tiles * p.t_tiles;
  const int64_t clusters = csize > 1 ? items : (items < sms ? items : sms);
  return launch_dependent(k, dim3((unsigned)(clusters * csize)), Cfg::kThreads, Cfg::smem_for(p.stages, p.kb_per_rank) + (p.own_sums ? (size_t)linear_sum_bytes(csize, p.M < NT ? p.M : NT) : 0), st,
                          csize, "linear_stream_kernel", tw, tx, p);
}

}  // namespace b200
