// Decode-sized block-FP8 GEMM (up to 32 rows of activations always, up to 256 where plan_gemm finds
// it the fastest): the roles of the operands are swapped so that the 128 weight rows of a tile fill
// the 128 lanes of the tensor-core tile and the few tokens are its N dimension:
//     D[n, m] = sum_k W[n, k] * X[m, k]        (UMMA M = 128 weight rows, N = NT tokens)
// A thread of the promotion warps then owns ONE weight row and NT (16 or 32) token
// accumulators instead of 128, so the per-K-block TMEM -> register promotion that bounds the
// large-tile kernel at small M shrinks 4-8x and the kernel streams the weights at HBM rate.
// Work item = (128-row weight tile, token tile, K split); one CTA per item, two CTAs per SM.
// K splits form a thread-block cluster (up to 8) who exchange their sums through distributed shared
// memory; a fan-out, and K too long for 8 splits, write fp32 partials that splitk_reduce_kernel sums.
#pragma once

#include "gemm_stream.cuh"

namespace b200 {

// Parameters are part of what a launch costs: 16 bytes more, 408 of them with the two tensor maps instead of 392, took every
// launch 0.12 us (9 x 2536 x 384, in a graph: 2.97 us, 3.08).
struct SkinnyParams {
  union {
    const float* As;  // As[m*as_sm + kb*as_sk]
    const void* x;    // QUANT: 16-bit activations [M, K], row-major
  };
  int64_t as_sm, as_sk;
  const float* Bs;  // [ceil(N/128)][num_kb]
  // packed power-of-two scales instead (As null): word (kb / 4) * ld + row holds the exponents of four K blocks; sfb_step rows
  // of words per 128 weight rows
  const int32_t *sfa, *sfb;
  int64_t sfa_ld, sfb_ld;
  int sfb_step;
  float eps;        // QUANT: least row-group maximum
  void* C;          // OutT [M, N], or fp32 partials [splits][M, N]
  int M, N, K, num_kb;
  int n_tiles, t_tiles, k_splits, kb_per_split;
  const uint8_t* w;  // the weights [N, K]
  int cluster;  // the K splits of an item are one cluster
  int* status;
};
static_assert(2 * sizeof(CUtensorMap) + sizeof(SkinnyParams) <= 392, "see above");

template <int NT, bool QUANT>
struct SkinnyCfg {
  static constexpr int kStages = 5;
  static constexpr int kStageW = 128 * kBK;  // 16 KB of weights
  static constexpr int kStageX = NT * kBK;   // 2 or 4 KB of activations
  static constexpr int kQuantRows = 8;  // QUANT: rows that the quantiser warps cover
  static constexpr int kQuantWarps = 4, kThreads = (QUANT ? 6 + kQuantWarps : 6) * 32;  // 4 promotion warps, producer, MMA issuer (, quantisers)
  // TMEM accumulator buffers: the tensor core runs this many K blocks ahead of the promotion warps, so the
  // commit -> tcgen05.ld -> arrive round trip (about a microsecond) is off the per-K-block path
  static constexpr int kAccBufs = 4;
  static constexpr int kTmemCols = kAccBufs * NT;
  static constexpr int kMaxKb = 64;          // K blocks one CTA may own (scales staged in smem)
  // sums exchanged within a cluster of K splits, [split][rows of this CTA][128]; with 32 tokens two CTAs per SM leave no
  // room for them and they go to the ring once it is idle
  static constexpr int kSumBytes = NT == 16 ? 21 * 512 : 0;
  static constexpr size_t kSmemBytes =
      (size_t)kStages * (kStageW + kStageX) + (size_t)kMaxKb * NT * 4 + kSumBytes + (QUANT ? kMaxKb * 8 : 0) + 1024 + 256;
};

// QUANT: X is the 16-bit input of a linear layer. Four more warps quantise the CTA's K range of its rows (same bytes and scales as
// the stand-alone quantiser), one K block after the other into the ring next to the weights, while those stream: quantiser and
// GEMM in one launch, the quantiser's time hidden behind the weights'. Bound by the weight stream and, between two calls, by the
// dependency wait, the first rows of x and the fill of the ring (3.7 us a projection). Prefetching more than three K blocks into
// L2 meanwhile makes it slower (1 row, four projections: 2 or 3 blocks 47.9, 5 49.7, 8 51.9 us).
template <int NT, bool QUANT, typename OutT>
__global__ void __launch_bounds__(SkinnyCfg<NT, QUANT>::kThreads, 2)
block_fp8_gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                             const SkinnyParams p) {
  using Cfg = SkinnyCfg<NT, QUANT>;
  constexpr int S = Cfg::kStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const uint32_t sW = smem_base;
  const uint32_t sX = smem_base + S * Cfg::kStageW;
  float* scales = reinterpret_cast<float*>(smem_al + (size_t)S * (Cfg::kStageW + Cfg::kStageX));  // [kb][NT]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(scales) + (size_t)Cfg::kMaxKb * NT * 4);
  const uint32_t bar0 = ptx::smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (S + s); };
  constexpr int NB = Cfg::kAccBufs;
  auto tfull_bar = [&](int b) { return bar0 + 8u * (2 * S + b); };
  auto tempty_bar = [&](int b) { return bar0 + 8u * (2 * S + NB + b); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * S + 2 * NB);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * S + 2 * NB + 1);
  // QUANT: scales of K block j are in the table (used once, behind the sums of the other splits)
  auto table_bar = [&](int j) { return bar0 + 256u + (uint32_t)Cfg::kSumBytes + 8u * j; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducerWarp = 4, kMmaWarp = 5;

  // work item
  const int item = blockIdx.x;
  const int ks = item % p.k_splits;
  const int tt = (item / p.k_splits) % p.t_tiles;
  const int nt = item / (p.k_splits * p.t_tiles);
  const int kb0 = ks * p.kb_per_split, kb1 = min(p.num_kb, kb0 + p.kb_per_split);
  const int n0 = nt * 128, m0 = tt * NT;
  // QUANT: rows that the 16 groups of eight lanes take side by side, 4 or 8; the other groups take the next K blocks. Four
  // K blocks at most are under way: with more than the ring's stages a group would wait for a phase of a stage's barrier that is
  // two ahead of it, which the parity does not tell from the one before.
  const int rows = min(NT, p.M - m0);
  const int q_rows = rows <= 4 ? 4 : Cfg::kQuantRows;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      ptx::mbar_init(full_bar(s), QUANT ? 1 + q_rows : 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < NB; ++b) {
      ptx::mbar_init(tfull_bar(b), 1);
      ptx::mbar_init(tempty_bar(b), 4);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
  }
  // a thread each; only waited for within the CTA, so __syncthreads below is all they need
  if (QUANT && threadIdx.x >= 32 && (int)threadIdx.x - 32 < kb1 - kb0) ptx::mbar_init(table_bar(threadIdx.x - 32), q_rows);
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
  if (p.cluster) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  // This grid is launched as a programmatic dependent: every operand, and at the end the output buffer, belongs to the
  // kernels before it in the stream, which may still run. The weight stream starts all the same, as a prefetch into L2
  // by the promotion warps, who have nothing else to do (a row each); after the wait they stage As[m, kb] * Bs[n0/128, kb]
  // for this item's tokens and K blocks in shared memory (their own 128-thread barrier: only they read the table).
  if (warp < 4) {
    if (n0 + (int)threadIdx.x < p.N)
      prefetch_weight_row(p.w + (int64_t)(n0 + threadIdx.x) * p.K + kb0 * kBK, min(kPrefetchKb, kb1 - kb0));
    grid_dependency_wait();
    const float* bs_row = p.Bs + (int64_t)nt * p.num_kb;
    for (int i = threadIdx.x; !QUANT && i < (kb1 - kb0) * NT; i += 128) {
      const int kb = kb0 + i / NT, t = i % NT;
      const int m = m0 + t;
      float s = 0.f;
      if (m < p.M) {
        if (p.As != nullptr) {
          s = __ldg(p.As + (int64_t)m * p.as_sm + (int64_t)kb * p.as_sk) * __ldg(bs_row + kb);
        } else {  // exponent byte -> power of two
          const uint32_t a = (uint32_t)__ldg(p.sfa + (kb >> 2) * p.sfa_ld + m) >> (8 * (kb & 3));
          const uint32_t b = (uint32_t)__ldg(p.sfb + (kb >> 2) * p.sfb_ld + (int64_t)nt * p.sfb_step) >> (8 * (kb & 3));
          s = __uint_as_float((a & 0xffu) << 23) * __uint_as_float((b & 0xffu) << 23);
        }
      }
      scales[i] = s;
    }
    if (!QUANT) asm volatile("bar.sync 1, 128;" ::: "memory");
  }

  float acc[NT];
  bool ok_sum = false;
  if (warp == kProducerWarp) {
    if (ptx::elect_one()) {
      bool ok = true;
      grid_dependency_wait();
      uint32_t it = 0;
      for (int kb = kb0; kb < kb1 && ok; ++kb, ++it) {
        const int s = it % S;
        ok = ptx::mbar_wait(empty_bar(s), ((it / S) & 1) ^ 1, abort_flag);
        if (!ok) break;
        ptx::mbar_expect_tx(full_bar(s), Cfg::kStageW + (QUANT ? 0 : Cfg::kStageX));
        ptx::tma_load_2d(sW + s * Cfg::kStageW, &tmap_w, kb * kBK, n0, full_bar(s));
        if (!QUANT) ptx::tma_load_2d(sX + s * Cfg::kStageX, &tmap_x, kb * kBK, m0, full_bar(s));
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    if (ptx::elect_one()) {
      constexpr uint32_t idesc = ptx::idesc_e4m3_f32(128, NT);
      bool ok = true;
      uint32_t it = 0;
      for (int kb = kb0; kb < kb1 && ok; ++kb, ++it) {
        const int s = it % S, b = it % NB;
        ok = ptx::mbar_wait(tempty_bar(b), ((it / NB) & 1) ^ 1, abort_flag) &&
             ptx::mbar_wait(full_bar(s), (it / S) & 1, abort_flag);
        if (!ok) break;
        ptx::tc_fence_after();
        const uint64_t dw = ptx::smem_desc_sw128(sW + s * Cfg::kStageW);
        const uint64_t dx = ptx::smem_desc_sw128(sX + s * Cfg::kStageX);
        const uint32_t d = tmem_base + b * NT;
#pragma unroll
        for (int k = 0; k < kBK / 32; ++k) ptx::mma_f8(d, dw + 2 * k, dx + 2 * k, idesc, k > 0);
        ptx::mma_commit(empty_bar(s));
        ptx::mma_commit(tfull_bar(b));
      }
    }
    __syncwarp();
  } else if (QUANT && warp > kMmaWarp) {
    if constexpr (QUANT) {
      // Eight lanes hold the 128 values of one (row, K block), 16 each; the groups of a warp have the same K block.
      static_assert(S >= 4, "the K blocks under way fit the ring");
      const int tid = threadIdx.x - (kMmaWarp + 1) * 32, chunk = tid & 7, row = (tid >> 3) & (q_rows - 1);
      const int step = 4 * Cfg::kQuantWarps / q_rows, first = (tid >> 3) / q_rows, nkb = kb1 - kb0;
      const unsigned group = 0xffu << (lane & 24);
      const OutT* src = static_cast<const OutT*>(p.x) + (int64_t)(m0 + min(row, rows - 1)) * p.K + (int64_t)kb0 * kBK + chunk * 16;
      const float* bs = p.Bs + (int64_t)nt * p.num_kb + kb0;
      constexpr int D = 4;  // K blocks in flight per group
      uint4 raw[D][2];
      float b[D];
      auto request = [&](int j, int u) {
        j = min(j, nkb - 1);
        raw[u][0] = ld_nc_16(src + (int64_t)j * kBK);
        raw[u][1] = ld_nc_16(src + (int64_t)j * kBK + 8);
        b[u] = __ldg(bs + j);
      };
      grid_dependency_wait();
#pragma unroll
      for (int u = 0; u < D; ++u) request(first + u * step, u);
      bool ok = true;
      for (int j0 = 0; j0 < nkb; j0 += D * step) {
#pragma unroll
        for (int u = 0; u < D; ++u) {
          if (j0 + u * step >= nkb) break;  // the same for the whole warp
          const int j = j0 + u * step + first;
          uint4 q;
          const float scale = quant_chunk<OutT>(raw[u], p.eps, q) * b[u];
          request(j + D * step, u);
          if (j >= nkb) continue;
          const int s = j % S;
          ok = ok && ptx::mbar_wait(empty_bar(s), ((j / S) & 1) ^ 1, abort_flag);
          if (ok && row < rows) {
            const uint32_t dst = sX + s * Cfg::kStageX + (row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w) : "memory");
            if (chunk == 0) scales[j * NT + row] = scale;
            ptx::fence_proxy_async_smem();  // generic-proxy writes -> the tensor core's reads
          }
          __syncwarp(group);
          if (ok && chunk == 0) {
            ptx::mbar_arrive(full_bar(s));
            ptx::mbar_arrive(table_bar(j));
          }
        }
      }
    }
  } else {
    // promotion warps: lane = weight row, columns = tokens
    const int n = n0 + warp * 32 + lane;
    const uint32_t lane_base = tmem_base + ((uint32_t)(warp * 32) << 16);
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t] = 0.f;
    bool ok = true;
    uint32_t it = 0;
    for (int kb = kb0; kb < kb1; ++kb, ++it) {
      const int b = it % NB;
      ok = ptx::mbar_wait(tfull_bar(b), (it / NB) & 1, abort_flag);
      if (QUANT) ok = ok && ptx::mbar_wait(table_bar(kb - kb0), 0, abort_flag);
      if (!ok) break;
      ptx::tc_fence_after();
      uint32_t v[32];
      if (NT == 32) {
        ptx::tmem_ld32(lane_base + b * NT, v);
        ptx::tmem_ld_wait(v);
      } else {
        ptx::tmem_ld16(lane_base + b * NT, v);
        ptx::tmem_ld_wait16(v);
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(tempty_bar(b));
      const float4* sc = reinterpret_cast<const float4*>(scales + (size_t)(kb - kb0) * NT);
#pragma unroll
      for (int j = 0; j < NT / 4; ++j) {
        const float4 s4 = sc[j];  // same address for every lane: broadcast
        acc[4 * j + 0] = fmaf(__uint_as_float(v[4 * j + 0]), s4.x, acc[4 * j + 0]);
        acc[4 * j + 1] = fmaf(__uint_as_float(v[4 * j + 1]), s4.y, acc[4 * j + 1]);
        acc[4 * j + 2] = fmaf(__uint_as_float(v[4 * j + 2]), s4.z, acc[4 * j + 2]);
        acc[4 * j + 3] = fmaf(__uint_as_float(v[4 * j + 3]), s4.w, acc[4 * j + 3]);
      }
    }
    ok_sum = ok;
    // The next kernels may start, as this grid drains. Signalled at the start they took their places while this grid still
    // ran, two CTAs on some SMs and none on others: four projections (6144..28672 x 4096..14336) in a graph, 1 / 16 rows,
    // 54.9 / 55.6 us, from here 50.9 / 54.3; of a rank of two 35.7 / 38.1 and 35.1 / 37.5.
    grid_launch_dependents();
    if (!p.cluster && ok && n < p.N) {
      OutT* out = static_cast<OutT*>(p.C) + (int64_t)ks * p.M * p.N + n;
#pragma unroll
      for (int t = 0; t < NT; ++t)
        if (m0 + t < p.M) out[(int64_t)(m0 + t) * p.N] = from_f32<OutT>(acc[t]);  // 32 lanes -> 32 consecutive n
    }
  }

  if (p.cluster) {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (Cfg::kSumBytes == 0) ptx::cluster_sync();  // every ring is idle
    // every split adds up its share of the rows: row t belongs to split t / per
    const int r = threadIdx.x & 127, per = (rows + p.k_splits - 1) / p.k_splits;
    const uint32_t sums_off = Cfg::kSumBytes ? (uint32_t)(reinterpret_cast<uint8_t*>(bars + 32) - smem_al) : 0u;
    if (warp < 4) {
      int owner = 0, j = 0;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        if (t < rows) ptx::st_cluster_f32(ptx::mapa(smem_base + sums_off, owner) + ((ks * per + j) * 128 + r) * 4, acc[t]);
        if (++j == per) j = 0, ++owner;
      }
    }
    __syncwarp();
    ptx::cluster_sync();
    if (warp < 4 && ok_sum && n0 + r < p.N) {
      const float* src = reinterpret_cast<const float*>(smem_al + sums_off) + r;
      OutT* out = static_cast<OutT*>(p.C) + n0 + r;
      const int t0 = ks * per, n_mine = min(per, rows - t0);
      constexpr int U = 4;  // rows in flight
      for (int j = 0; j < n_mine; j += U) {
        float sum[U];
#pragma unroll
        for (int u = 0; u < U; ++u) sum[u] = 0.f;
        for (int c = 0; c < p.k_splits; ++c)  // split order: the same sum on every run
#pragma unroll
          for (int u = 0; u < U; ++u) sum[u] += src[(c * per + min(j + u, n_mine - 1)) * 128];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (j + u < n_mine) out[(int64_t)(m0 + t0 + j + u) * p.N] = from_f32<OutT>(sum[u]);
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

// Number of K splits for the skinny kernel: about two work items per SM, each with at least
// two K blocks and at most kMaxKb.
inline int skinny_k_splits(int64_t M, int64_t N, int64_t K, int nt, int sms) {
  const int64_t items = cdiv(N, 128) * cdiv(M, nt);
  const int64_t num_kb = cdiv(K, 128);
  int64_t s = (2 * (int64_t)sms) / items;
  if (s > num_kb / 2) s = num_kb / 2;
  if (s < 1) s = 1;
  const int64_t need = cdiv(num_kb, 64);  // a CTA stages the scales of at most 64 K blocks
  if (s < need) s = need;
  if (s > 16) s = 16 > need ? 16 : need;
  return (int)s;
}

inline int skinny_token_tile(int64_t M) { return M <= 16 ? 16 : 32; }

// K splits as one cluster, no empty one; 1: through memory. Clusters of up to 4 fit the chip's SM groups anywhere, of up to 6 or
// 8 where few items leave most of the chip free, and none may have to wait for a second wave: 96 items in clusters of 3 fill
// 288 of the 296 slots, not all of them usable (50 x 6144 x 4096: 18.4 us against 11.5). With 32 tokens the exchange needs the
// idle ring and only pays from three splits on. 16 x 4096 x 4096: 10.0 -> 7.3 us, 16 x 1280 x 8192: 9.0 -> 6.5,
// 32 x 1536 x 4096: 9.4 -> 6.8.
inline int skinny_cluster(int64_t items, int64_t K, int nt, int want) {
  const int64_t num_kb = cdiv(K, 128);
  const int cap = items * 8 <= 96 ? 8 : items * 6 <= 128 ? 6 : 4;
  int c = want < cap ? want : cap;
  c = (int)cdiv(num_kb, cdiv(num_kb, c));
  if (cdiv(num_kb, c) > 64 || items * c > 264 || (nt > 16 && c < 3)) return 1;
  return c;
}

template <int NT, bool QUANT, typename OutT>
inline int launch_skinny_inst(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, cudaStream_t st) {
  auto k = block_fp8_gemm_skinny_kernel<NT, QUANT, OutT>;
  const size_t smem = SkinnyCfg<NT, QUANT>::kSmemBytes;
  if (int rc_smem = allow_smem(k, smem, "GEMM kernel")) return rc_smem;
  // programmatic dependent of the kernel before it (normally the activation quantiser, which
  // signals launch_dependents at once): set-up and the first weight prefetches overlap its tail
  return launch_dependent(k, dim3((unsigned)(p.n_tiles * p.t_tiles * p.k_splits)), SkinnyCfg<NT, QUANT>::kThreads, smem, st,
                          p.cluster ? p.k_splits : 1, "block_fp8_gemm_skinny_kernel", tw, tx, p);
}

// out: OutT [M, N] when splits == 1 or they are a cluster, else fp32 partials [splits][M, N]. X null: p.x is quantised.
template <typename OutT>
inline int launch_skinny(const void* X, const void* W, SkinnyParams p, int splits, bool cluster, cudaStream_t st) {
  constexpr int kQuantRows = SkinnyCfg<16, true>::kQuantRows;
  B200_UNSUPPORTED(X == nullptr && (p.M > kQuantRows || sizeof(OutT) != 2),
                   "gemm: the decode kernel quantises %d rows of 16-bit input at most, not %d", kQuantRows, p.M);
  const int nt = skinny_token_tile(p.M);
  p.num_kb = (int)cdiv(p.K, kBK);
  p.n_tiles = (int)cdiv(p.N, 128);
  p.t_tiles = (int)cdiv(p.M, nt);
  p.k_splits = splits;
  p.kb_per_split = (int)cdiv(p.num_kb, splits);
  p.cluster = cluster;
  p.w = static_cast<const uint8_t*>(W);
  p.status = device_status_word();
  if (!p.status) {
    set_error_detail("cannot resolve the device status word");
    return B200_E_LAUNCH;
  }
  CUtensorMap tw, tx;
  int rc = make_tmap_u8(&tw, W, (uint64_t)p.N, (uint64_t)p.K, 128, "W");
  if (rc) return rc;
  if constexpr (sizeof(OutT) == 2) {
    if (X == nullptr) return launch_skinny_inst<16, true, OutT>(tw, tw, p, st);
  }
  rc = make_tmap_u8(&tx, X, (uint64_t)p.M, (uint64_t)p.K, (uint32_t)nt, "X");
  if (rc) return rc;
  if (nt == 16) return launch_skinny_inst<16, false, OutT>(tw, tx, p, st);
  return launch_skinny_inst<32, false, OutT>(tw, tx, p, st);
}

}  // namespace b200
