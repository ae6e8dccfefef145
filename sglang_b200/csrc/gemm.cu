// w8a8_block_fp8_matmul: dense block-FP8 GEMM entry point (tcgen05 / TMEM / TMA kernel in
// gemm_kernel.cuh).
#include "gemm_host.cuh"
#include "gemm_pair.cuh"
#include "gemm_skinny.cuh"
#include "linear_stream.cuh"
#include "gemm_ue8m0.cuh"
#include "gemm_ue8m0_pair.cuh"

namespace b200 {

// Destinations of a fan-out GEMM (see GemmParams::n_dest): n == 0 means "C only".
struct FanOut {
  int n, by_tile;
  void* dest[kMaxFan];
};

// C[m, n] = sum over splits of the fp32 partials; 8 elements per thread. With a fan-out the sum
// goes to every destination buffer (or to the owner of the 128-row block) instead of C.
template <typename OutT>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ partial, OutT* __restrict__ C,
                                                            int64_t mn, int splits, const FanOut fan, int64_t N) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  // launched with programmatic stream serialisation: this grid may start while the GEMM that
  // writes the partials is still draining; everything above is index arithmetic only
  grid_launch_dependents();
  grid_dependency_wait();
  if (i >= mn) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int s = 0; s < splits; ++s) {
    const float4 a = *reinterpret_cast<const float4*>(partial + (int64_t)s * mn + i);
    const float4 b = *reinterpret_cast<const float4*>(partial + (int64_t)s * mn + i + 4);
    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
    acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
  }
  if (fan.n == 0) {
    store8<OutT>(C + i, acc);
    return;
  }
  const int d0 = fan.by_tile ? (int)((i / N / kBM) % fan.n) : 0;
  const int d1 = fan.by_tile ? d0 + 1 : fan.n;
  for (int d = d0; d < d1; ++d) store8<OutT>(static_cast<OutT*>(fan.dest[d]) + i, acc);
}

template <typename OutT>
static int launch_reduce(const float* partial, void* C, int64_t mn, int splits, cudaStream_t st,
                         const FanOut& fan = FanOut{}, int64_t N = 1) {
  // Programmatic dependent launch: the grid is set up while the producing GEMM finishes (the decode
  // kernel signals launch_dependents once all its CTAs run); griddepcontrol.wait in the kernel holds
  // it until the partials are complete and visible.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cdiv(mn, 8 * 256));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, splitk_reduce_kernel<OutT>, partial, static_cast<OutT*>(C), mn, splits, fan, N);
  if (e != cudaSuccess) {
    set_error_detail("splitk_reduce_kernel: %s", cudaGetErrorString(e));
    return B200_E_LAUNCH;
  }
  return check_launch("splitk_reduce_kernel");
}

}  // namespace b200

namespace b200 {
constexpr int64_t kSkinnyMaxM = 32;       // rows up to which the swapped-operand decode kernel is always used
constexpr int64_t kSkinnyPlanMaxM = 256;  // ... and up to which it is considered
struct GemmPlan {
  int splits;   // K splits (fp32 partials + a reduction pass when > 1)
  int pair_bn;  // 0: single-CTA 128 x 256 tiles, else CTA pairs with 256 x pair_bn tiles
  bool skinny;  // swapped-operand decode kernel
  bool stream;  // weight-streaming kernel, token tiles of 64
  bool csum;    // the K splits of a pair's tile are one cluster and summed there
  double us;    // modelled time (0: not modelled, decode sizes)
};

// K splits of the decode kernel (gemm_skinny.cuh) when `splits` are asked for, and whether they are summed within clusters.
struct SkinnySplit {
  int splits;
  bool cluster;
  bool direct() const { return splits == 1 || cluster; }  // the kernel writes the result itself, without partials in memory
};
static SkinnySplit skinny_split(int64_t M, int64_t N, int64_t K, int splits) {
  while (cdiv(cdiv(K, 128), splits) > SkinnyCfg<16, false>::kMaxKb) ++splits;  // scales of one item fit its smem table
  const int nt = skinny_token_tile(M);
  const int cluster = splits > 1 && tuning().gemm_splitk <= 0 ? skinny_cluster(cdiv(N, 128) * cdiv(M, nt), K, nt, splits) : 1;
  return cluster > 1 ? SkinnySplit{cluster, true} : SkinnySplit{splits, false};
}

// Modelled time of the decode kernel. Its CTAs run two to an SM: one that has its SM to itself takes 0.22 us per 128-K block, one
// that shares it 0.39. More CTAs than places are partly whole waves and partly fill in as others end (long K ranges drift apart);
// nothing is faster than the weights from memory (5.4 TB/s; 4.4 where they nearly fill the L2, which the next token tile then misses:
// 64 x 8192 x 7168 16.0 us, x 14336 31.3) or, once per 32 rows, from L2 (12.5 TB/s). Over 450 sizes of 34 to 256
// rows it is within 5 % on average; a rate per byte alone (9.5 TB/s) was 12 % off, most of it where K is short:
// 65..128 x 8192 x 512 4.3 us, 8.5 modelled, so the plan took pairs at 5.4.
static double skinny_us(int64_t M, int64_t N, int64_t K, int sms, SkinnySplit s, double sum) {
  const int64_t t_tiles = cdiv(M, skinny_token_tile(M)), ctas = cdiv(N, 128) * t_tiles * s.splits;
  const double kb = (double)cdiv(cdiv(K, 128), s.splits), places = 2.0 * sms, waves = (double)cdiv(ctas, 2 * sms);
  double work = ctas <= sms ? kb * 0.222 : kb * 0.389;
  if (waves > 1.0) work = kb * 0.389 * (0.56 * waves + 0.44 * (double)ctas / places) + 2.6 * (waves - 1.0);
  const double memory = (double)N * (double)K / (N * K > (96 << 20) ? 4.4e6 : 5.4e6), l2 = (double)t_tiles * (double)N * (double)K / 12.5e6;
  if (work < memory) work = memory;
  if (work < l2) work = l2;
  return 2.67 + work + sum;
}
static double skinny_us(int64_t M, int64_t N, int64_t K, int sms, SkinnySplit s) {
  const double sum = s.splits == 1 ? 0.0 : s.cluster ? 2.0 : 0.78 + 1.52 * s.splits * (double)M * (double)N / 1e6;
  return skinny_us(M, N, K, sms, s, sum);
}

// SMs that plans are made for
static int plan_sms() { return sm_count() < 148 ? sm_count() : 148; }

// Kernel, tile and K split of a dense problem: the one whose modelled time is least. The model is launch and set-up, then
// whole waves of tiles, each its 128-K blocks and an epilogue; nothing is faster than reading the weights (6.2 TB/s). Where the
// tiles of 128-wide pairs leave half of the chip idle their K range is split 2 or 4 ways within clusters, of which this part holds
// 33 and 15 at once; the sum costs 2 to 3 us. The constants are fits to every kernel's time at 632 sizes, 16 weight shapes (1280..28672
// x 1024..14336) times 17 row counts (33..2200) and as many spread over 17..2200 x 136..16384 x 256..16384: the plan is
// 0.4 % behind the best kernel on average up to 256 rows, 1 % over all (at the power cap repeats of one kernel differ by more). E.g. 203 x 4096 x 4096: decode kernel 14.1 us, pairs 128 wide 12.5, their K split two ways
// 10.3; 203 x 4096 x 14336: 24.5 with partials through memory, 19.7; 512 x 1280 x 8192 16.6 and 13.9.
//
// A fan-out (its result goes to several buffers) is planned from what can do that: the 8-warp tile kernel unsplit, or the decode
// and 16-warp kernels with fp32 partials, whose reduction pass writes to the buffers (1.5 us and 4.5 us per million partials; no
// clusters, no weight streaming). Fitted to 567 sizes of 33..1200 rows with the buffers on this GPU, 0.5 % behind the best;
// e.g. 72 x 6144 x 4096: decode kernel 11.4 us, tile kernel unsplit 22.2; 300 x 4096 x 14336: unsplit 64, 2 splits of 128-wide
// pairs 35; 112 x 5120 x 1536: 8.7 and 11.8.
struct PlanFor {
  bool fanout = false;
  double unpack_us = 0.0;  // what every kernel but the decode kernel waits for first (packed scales, which that one reads itself)
};
static GemmPlan plan_gemm(int64_t M, int64_t N, int64_t K, int sms, bool may_pair, PlanFor use = {}) {
  const Tuning& tune = tuning();
  const int64_t num_kb = cdiv(K, 128);
  const int64_t skinny_max = tune.gemm_skinny_max_m >= 0 ? tune.gemm_skinny_max_m : kSkinnyMaxM;
  const bool skinny_ok = may_pair && tune.gemm_skinny != 0;
  if (may_pair && tune.gemm_stream > 0) return {1, 0, false, true, false, 0.0};
  if (M <= skinny_max && skinny_ok) return {skinny_k_splits(M, N, K, skinny_token_tile(M), sms), 0, true, false, false, 0.0};
  if (may_pair && (tune.gemm_2cta == 1282 || tune.gemm_2cta == 1284) && N >= 256) return {(int)tune.gemm_2cta % 10, 128, false, false, true, 0.0};
  if (may_pair && tune.gemm_2cta > 0 && N >= 256) return {1, tune.gemm_2cta == 1 ? 256 : tune.gemm_2cta == 2 ? 0 : (int)tune.gemm_2cta, false, false, false, 0.0};
  GemmPlan best = {1, 0, false, false, false, 1e30};  // its time without unpacking
  const double stream_us = (double)N * (double)K / 6.2e6;
  // K splits through memory: a reduction pass and the fp32 partials, written and read at about 2 TB/s
  auto memory_sum = [&](int s) {
    const double partials = s * (double)M * (double)N / 1e6;
    return use.fanout ? 1.5 + 4.5 * partials : N <= 128 ? 2.2 + 2.3 * partials : 3.6 + 2.6 * partials;
  };
  // crowd: what tiles side by side cost one another when every slot has one (256 x 4096 x 1024, 32 pairs, 5.4 us; 64 x 8192 x 1024, 64
  // pairs, 7.1)
  auto consider = [&](int bm, int bn, int slots, double base, double us_per_kb, double epilogue, double crowd, int pair_bn, int first,
                      int last) {
    const int64_t tiles = cdiv(M, bm) * cdiv(N, bn);
    const double busy = tiles < slots ? (double)tiles / slots : 1.0;
    for (int s = 1; s <= last && (s == 1 || num_kb >= 4 * s); ++s) {
      const double waves = (double)cdiv(tiles * s, slots);
      double work = waves * ((double)cdiv(num_kb, s) * us_per_kb + epilogue);
      if (work < stream_us) work = stream_us;
      const double us = base + crowd * busy + work + (s > 1 ? memory_sum(s) : 0.0);
      if (s >= first && us < best.us) best = {s, pair_bn, false, false, false, us};
      if (tiles * s >= slots) break;  // every slot is busy: more splits only add partials
    }
  };
  const bool pairs = may_pair && tune.gemm_2cta != 0 && N >= 256 && sms >= 2;
  if (use.fanout) {
    if (N >= 256) consider(128, 256, sms, 4.0, 0.64, 1.5, 0.0, 0, 1, 1);
    else if (N > 128) consider(128, 256, sms, 3.7, 0.45, 1.5, 0.0, 0, 1, 1);
    else consider(128, 128, sms, 3.7, 0.30, 0.5, 0.0, 0, 1, 1);
    consider(128, N > 128 ? 256 : 128, sms, 3.5, 0.55, 1.0, 0.0, 0, 2, 8);
    if (pairs) consider(256, 128, sms / 2, 3.8, 0.225, 0.85, 0.0, 128, 2, 8);
  } else {
    // Splits of pairs go through memory on partitions of the part only: all of it sums them in clusters (below), whose numbers at
    // once are known for 148 SMs.
    const int max_splits = pairs && sms >= 148 ? 1 : 8;
    if (N >= 256) {
      consider(128, 256, sms, 3.5, 0.44, 1.0, 0.0, 0, 1, max_splits);
    } else if (N > 128) {  // 502 x 192 x 1536: unsplit 7.8 us, three splits 11.5, which the costs of the line above would take
      consider(128, 256, sms, 3.1, 0.35, 0.7, 0.0, 0, 1, max_splits);
    } else {
      consider(128, 128, sms, 3.1, 0.27, 0.05, 0.0, 0, 1, max_splits);
    }
    if (pairs) {
      consider(256, 256, sms / 2, 3.5, 0.38, 1.8, 0.0, 256, 1, max_splits);
      consider(256, 192, sms / 2, 4.25, 0.35, 1.2, 0.0, 192, 1, max_splits);
      consider(256, 128, sms / 2, 3.1, 0.225, 0.85, 1.0, 128, 1, max_splits);
    }
  }
  if (pairs && !use.fanout && sms >= 148) {
    const int64_t tiles = cdiv(M, 256) * cdiv(N, 128);
    for (int s = 2; s <= 4; s += 2) {
      if (tiles > (s == 2 ? 33 : 15) || num_kb < 4 * s) continue;
      double work = (double)cdiv(num_kb, s) * (s == 2 ? 0.21 : 0.18);
      if (work < stream_us) work = stream_us;
      const double us = (s == 2 ? 5.2 + 1.5 * (double)(2 * tiles) / 74.0 : 7.4) + work;
      if (us < best.us) best = {s, 128, false, false, true, us};
    }
  }
  if (may_pair && !use.fanout && tune.gemm_stream != 0 && M > 32 && M <= 128) {
    int csize, kb, stages, own;
    if (plan_linear_stream<64, false>(M, N, K, sms, csize, kb, stages, own)) {
      // 0.44 us per 128-K block of 256 weight rows x 64 tokens; a cluster's sum costs a microsecond more, and clusters fill 132 of
      // 148 SMs at most (80 x 6144 x 4096 in clusters of 3: 24.8 us, two waves)
      const int64_t items = cdiv(N, 256) * cdiv(M, 64);
      double work = (double)cdiv(items * csize, csize > 1 && sms >= 148 ? sms - 16 : sms) * kb * 0.44;
      if (work < (double)N * (double)K / 6.4e6) work = (double)N * (double)K / 6.4e6;
      const double us = 7.5 + (csize > 1 ? 1.0 : 0.0) + work;
      if (us < best.us) best = {1, 0, false, true, false, us};
    }
  }
  if (skinny_ok && M <= (tune.gemm_skinny_max_m >= 0 ? skinny_max : kSkinnyPlanMaxM)) {
    const int splits = skinny_k_splits(M, N, K, skinny_token_tile(M), sms);
    const SkinnySplit split = skinny_split(M, N, K, splits);
    double us = use.fanout ? skinny_us(M, N, K, sms, split, 0.0) + 1.2 + 1.27 * split.splits * (double)M * (double)N / 1e6
                           : skinny_us(M, N, K, sms, split);
    // packed words are staged by each CTA before its first sum: 64 x 14336 x 8192, 64 K blocks, 35 us (30 on fp32 scales)
    if (use.unpack_us > 0.0) us += 0.02 * (double)cdiv(num_kb, split.splits);
    if (us < best.us + use.unpack_us) best = {splits, 0, true, false, false, us};
  }
  if (!best.skinny) best.us += use.unpack_us;
  return best;
}
}

namespace b200 {
// fp32 partials of the split that this device's SMs pick, 148 without a device (or the tuning knobs force)
static size_t partial_bytes(int64_t M, int64_t N, int64_t K, PlanFor use = {}) {
  const Tuning& tune = tuning();
  const GemmPlan plan = plan_gemm(M, N, K, plan_sms(), tune.gemm_bn < 0, use);
  int s = plan.csum && !use.fanout ? 1 : plan.splits;  // summed in clusters
  if (tune.gemm_splitk > s) s = (int)tune.gemm_splitk;
  if (tune.gemm_skinny_max_m >= 0 && s < 16) s = 16;
  return s > 1 ? (size_t)s * (size_t)M * (size_t)N * sizeof(float) : 0;
}
}  // namespace b200

extern "C" size_t b200_w8a8_block_fp8_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  return M <= 0 || N <= 0 || K <= 0 ? 0 : b200::partial_bytes(M, N, K);
}

namespace b200 {
// What a dense problem runs: kernel, columns of its tile, K splits and where they are summed (the codes of b200_plan_dense).
// gemm_impl and the linear layer launch it, b200_plan_dense reports it.
struct GemmRoute {
  int kernel, tile_n, splits, sum;
};
static GemmRoute skinny_route(int64_t M, int64_t N, int64_t K, int splits, bool fanout, int kernel) {
  // a fan-out takes the same splits through memory, so its sums are those of the plain GEMM where that runs the decode kernel too
  const SkinnySplit s = skinny_split(M, N, K, splits);
  return {kernel, 128, s.splits, s.direct() && !fanout ? (s.splits > 1 ? B200_SUM_CLUSTER : B200_SUM_NONE) : B200_SUM_MEMORY};
}
static GemmRoute route_gemm(int64_t M, int64_t N, int64_t K, int sms, PlanFor use = {}) {
  const Tuning& tune = tuning();
  const int force_bn = tune.gemm_bn == 128 || tune.gemm_bn == 256 ? (int)tune.gemm_bn : 0;
  const GemmPlan plan = plan_gemm(M, N, K, sms, force_bn == 0, use);
  int splits = plan.splits;
  if (tune.gemm_splitk > 0) splits = (int)tune.gemm_splitk;
  if (splits > (int)cdiv(K, 128)) splits = (int)cdiv(K, 128);
  if (plan.stream && !use.fanout && tune.gemm_splitk <= 0) {
    int csize = 1, kb, stages, own;
    plan_linear_stream<64, false>(M, N, K, sms, csize, kb, stages, own);
    return {B200_KERNEL_STREAM, 256, csize, csize > 1 ? B200_SUM_CLUSTER : B200_SUM_NONE};
  }
  if (plan.skinny) return skinny_route(M, N, K, splits, use.fanout, B200_KERNEL_SKINNY);
  // the 8-warp tile kernel keeps the 128-wide tile (N <= 128) and the fan-out epilogue
  const bool wide = force_bn == 0 && N > 128 && tune.gemm_2cta != 0;
  // as many splits as the cluster has pairs, some of them empty where K has fewer blocks
  if (plan.csum && wide && !use.fanout && tune.gemm_splitk <= 0) return {B200_KERNEL_WIDE, plan.pair_bn, plan.splits, B200_SUM_CLUSTER};
  const int sum = splits > 1 ? B200_SUM_MEMORY : B200_SUM_NONE;
  if (wide && (splits > 1 || !use.fanout)) return {B200_KERNEL_WIDE, plan.pair_bn, splits, sum};
  return {B200_KERNEL_TILE, force_bn, splits, sum};
}

// The decode kernel as skinny_route laid it out; sp holds the scales (or the input to quantise).
static int run_skinny(const void* A, const void* B, SkinnyParams sp, const GemmRoute& r, void* C, int c_dtype, int64_t M, int64_t N,
                      int64_t K, void* workspace, size_t workspace_bytes, cudaStream_t st, const FanOut& fan) {
  sp.M = (int)M; sp.N = (int)N; sp.K = (int)K;
  const int splits = r.splits;
  if (r.sum != B200_SUM_MEMORY) {
    sp.C = C;
    if (c_dtype == B200_BF16) return launch_skinny<__nv_bfloat16>(A, B, sp, splits, splits > 1, st);
    if (c_dtype == B200_F16) return launch_skinny<__half>(A, B, sp, splits, splits > 1, st);
    return launch_skinny<float>(A, B, sp, splits, splits > 1, st);
  }
  const size_t need = (size_t)splits * (size_t)M * (size_t)N * sizeof(float);
  if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 15) != 0) {
    set_error_detail("gemm: split-K needs a 16-byte aligned workspace of %zu bytes (got %zu)", need, workspace_bytes);
    return B200_E_WORKSPACE;
  }
  sp.C = workspace;
  int rc = launch_skinny<float>(A, B, sp, splits, false, st);
  if (rc) return rc;
  const float* part = static_cast<const float*>(workspace);
  if (c_dtype == B200_BF16) return launch_reduce<__nv_bfloat16>(part, C, M * N, splits, st, fan, N);
  if (c_dtype == B200_F16) return launch_reduce<__half>(part, C, M * N, splits, st, fan, N);
  return launch_reduce<float>(part, C, M * N, splits, st, fan, N);
}

static int gemm_impl(const void* A, const float* As, int64_t as_stride_m, int64_t as_stride_k, const void* B,
                     const float* Bs, void* C, int c_dtype, int64_t M, int64_t N, int64_t K, void* workspace,
                     size_t workspace_bytes, void* stream, const FanOut& fan) {
  B200_CHECK_ARG(M >= 0 && N >= 0 && K >= 0, "gemm: negative shape");
  if (M == 0 || N == 0) return B200_OK;
  B200_CHECK_ARG(K > 0, "gemm: K must be positive");
  B200_CHECK_ARG(A && As && B && Bs && (C || fan.n > 0), "gemm: null pointer");
  B200_CHECK_ARG(((uintptr_t)A & 15) == 0 && ((uintptr_t)B & 15) == 0 && ((uintptr_t)C & 15) == 0,
                 "gemm: A, B and C must be 16-byte aligned");
  for (int d = 0; d < fan.n; ++d)
    B200_CHECK_ARG(fan.dest[d] && ((uintptr_t)fan.dest[d] & 15) == 0, "gemm: fan-out destination %d null or unaligned", d);
  B200_UNSUPPORTED(K % 16 != 0, "gemm: K=%lld must be a multiple of 16 (TMA row pitch)", (long long)K);
  B200_UNSUPPORTED(M > 0x7fffff00LL || N > 0x7fffff00LL || K > 0x7fffff00LL, "gemm: dimension too large");
  B200_UNSUPPORTED(N % 8 != 0, "gemm: N=%lld must be a multiple of 8 (vector stores)", (long long)N);
  GemmParams p = {};
  p.As = As; p.as_sm = as_stride_m; p.as_sk = as_stride_k;
  p.Bs = Bs; p.C = C; p.ldc = N;
  p.M = (int)M; p.N = (int)N; p.K = (int)K;
  p.n_dest = fan.n; p.dest_by_tile = fan.by_tile;
  for (int d = 0; d < fan.n; ++d) p.dest[d] = fan.dest[d];
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  B200_CHECK_ARG(c_dtype == B200_BF16 || c_dtype == B200_F16 || c_dtype == B200_F32, "gemm: unknown output dtype code %d",
                 c_dtype);
  const GemmRoute r = route_gemm(M, N, K, plan_sms(), PlanFor{fan.n > 0});
  const int splits = r.splits, bn = r.tile_n;
  if (r.kernel == B200_KERNEL_STREAM) {
    LinearStreamParams lp = {};
    lp.As = As; lp.as_sm = as_stride_m; lp.as_sk = as_stride_k; lp.Bs = Bs; lp.out = C;
    lp.M = (int)M; lp.N = (int)N; lp.K = (int)K;
    if (c_dtype == B200_BF16) return launch_linear_stream<64, false, __nv_bfloat16>(B, A, lp, st);
    if (c_dtype == B200_F16) return launch_linear_stream<64, false, __half>(B, A, lp, st);
    return launch_linear_stream<64, false, float>(B, A, lp, st);
  }
  if (r.kernel == B200_KERNEL_SKINNY) {
    SkinnyParams sp = {};
    sp.As = As; sp.as_sm = as_stride_m; sp.as_sk = as_stride_k; sp.Bs = Bs;
    return run_skinny(A, B, sp, r, C, c_dtype, M, N, K, workspace, workspace_bytes, st, fan);
  }
  const bool wide = r.kernel == B200_KERNEL_WIDE;
  if (r.sum == B200_SUM_CLUSTER) {
    if (c_dtype == B200_BF16) return launch_gemm_wide<__nv_bfloat16>(bn, A, B, p, splits, true, st);
    if (c_dtype == B200_F16) return launch_gemm_wide<__half>(bn, A, B, p, splits, true, st);
    return launch_gemm_wide<float>(bn, A, B, p, splits, true, st);
  }
  if (splits > 1) {
    // few tiles: fp32 partials per K split in the workspace, then one reduction pass
    const size_t need = (size_t)splits * (size_t)M * (size_t)N * sizeof(float);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 15) != 0) {
      set_error_detail("gemm: split-K needs a 16-byte aligned workspace of %zu bytes (got %zu)", need, workspace_bytes);
      return B200_E_WORKSPACE;
    }
    p.C = workspace;
    p.split_stride = M * N;
    p.n_dest = 0;  // the partials stay local; the reduction pass fans the sum out
    int rc = wide ? launch_gemm_wide<float>(bn, A, B, p, splits, false, st)
                  : launch_gemm<GEMM_DENSE, float>(A, B, N, p, bn, st, splits);
    if (rc) return rc;
    const float* part = static_cast<const float*>(workspace);
    if (c_dtype == B200_BF16) return launch_reduce<__nv_bfloat16>(part, C, M * N, splits, st, fan, N);
    if (c_dtype == B200_F16) return launch_reduce<__half>(part, C, M * N, splits, st, fan, N);
    return launch_reduce<float>(part, C, M * N, splits, st, fan, N);
  }
  if (wide) {
    if (c_dtype == B200_BF16) return launch_gemm_wide<__nv_bfloat16>(bn, A, B, p, 1, false, st);
    if (c_dtype == B200_F16) return launch_gemm_wide<__half>(bn, A, B, p, 1, false, st);
    return launch_gemm_wide<float>(bn, A, B, p, 1, false, st);
  }
  switch (c_dtype) {
    case B200_BF16: return launch_gemm<GEMM_DENSE, __nv_bfloat16>(A, B, N, p, bn, st);
    case B200_F16: return launch_gemm<GEMM_DENSE, __half>(A, B, N, p, bn, st);
    default: return launch_gemm<GEMM_DENSE, float>(A, B, N, p, bn, st);
  }
}
}  // namespace b200

extern "C" int b200_w8a8_block_fp8_gemm(const void* A, const float* As, int64_t as_stride_m, int64_t as_stride_k,
                                        const void* B, const float* Bs, void* C, int c_dtype, int64_t M, int64_t N,
                                        int64_t K, void* workspace, size_t workspace_bytes, void* stream) {
  return b200::gemm_impl(A, As, as_stride_m, as_stride_k, B, Bs, C, c_dtype, M, N, K, workspace, workspace_bytes, stream,
                         b200::FanOut{});
}

extern "C" size_t b200_w8a8_block_fp8_gemm_fanout_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const size_t partials = b200::partial_bytes(M, N, K, b200::PlanFor{true});
  // the decode kernel always goes through an fp32 partial when its result is fanned out
  const size_t one = M <= b200::kSkinnyPlanMaxM ? (size_t)M * (size_t)N * sizeof(float) : 0;
  return partials > one ? partials : one;
}

extern "C" int b200_w8a8_block_fp8_gemm_fanout(const void* A, const float* As, int64_t as_stride_m, int64_t as_stride_k,
                                               const void* B, const float* Bs, void* const* dest, int n_dest,
                                               int dest_by_tile, int c_dtype, int64_t M, int64_t N, int64_t K,
                                               void* workspace, size_t workspace_bytes, void* stream) {
  using namespace b200;
  B200_CHECK_ARG(dest != nullptr && n_dest >= 1 && n_dest <= kMaxFan, "gemm fan-out: %d destinations (1..%d)", n_dest,
                 kMaxFan);
  FanOut fan = {};
  fan.n = n_dest;
  fan.by_tile = dest_by_tile != 0;
  for (int d = 0; d < n_dest; ++d) fan.dest[d] = dest[d];
  return gemm_impl(A, As, as_stride_m, as_stride_k, B, Bs, nullptr, c_dtype, M, N, K, workspace, workspace_bytes, stream,
                   fan);
}

// Quantised activations of a linear layer: FP8 rows, then column-major scales, in front of the GEMM's own workspace.
namespace b200 {
static int run_linear_stream(const void* x, int x_dtype, const void* B, const float* Bs, void* out, int64_t M, int64_t N, int64_t K,
                             float eps, cudaStream_t st) {
  LinearStreamParams p = {};
  p.x = x; p.Bs = Bs; p.out = out; p.M = (int)M; p.N = (int)N; p.K = (int)K; p.eps = eps;
  return x_dtype == B200_BF16 ? launch_linear_stream<16, true, __nv_bfloat16>(B, nullptr, p, st)
                               : launch_linear_stream<16, true, __half>(B, nullptr, p, st);
}
static size_t linear_q_bytes(int64_t M, int64_t K) { return align_up((size_t)(M * K), 256); }
static size_t linear_s_bytes(int64_t M, int64_t K) { return align_up((size_t)(M * (K / 128)) * 4, 256); }
// One launch (linear_stream.cuh) or quantiser + GEMM. The one launch saves the quantiser's and the reduction's, but every
// CTA quantises its K range of x for itself. On the GPU the two are level within a few tenths of a microsecond up to 32 (row,
// K block) groups per CTA (1 x 1536 x 4096: 4.7 us against 5.2, 1 x 4096 x 1792: 5.3 against 4.9) and the second wins beyond
// (16 x 768 x 4096: 6.6 against 5.2) and for larger weights (1 x 8192 x 3584: 8.3 against 7.2); with small weights the GPU
// finishes before the host, which pays 4.7 us for one launch and 7 for two.
constexpr int64_t kLinearStreamMaxM = 16;
static bool linear_one_launch(int64_t M, int64_t N, int64_t K, int sms, int* ranks = nullptr) {
  int csize, kb, stages, own;
  if (M > kLinearStreamMaxM || tuning().linear_decode_fused == 0 || tuning().linear_decode_fused == 2 ||
      !plan_linear_stream<16, true>(M, N, K, sms, csize, kb, stages, own) ||
      kb * M > 32 || N * K >= (16 << 20))
    return false;
  if (ranks) *ranks = csize;
  return true;
}
// Quantiser inside the decode GEMM (one launch): up to 8 rows, where the plan takes that kernel and its splits are summed
// within clusters, and where every CTA's share of the quantising hides behind its weights. It does while no two CTAs share an SM
// (clusters fill 132 of 148): 4096 x 4096, 1 row, called one by one 6.5 us against 7.6 with a launch of its own (in a graph
// 6.5 and 6.6), 4096 x 14336 13.0 and 14.2 (13.4).
// A few SMs with two CTAs hold all others up (160 CTAs, 8 x 5120 x 5120 10.1 and 9.0; 144, 8 x 4608 x 7168 11.4 and 10.2), and short K
// ranges leave nothing to hide behind (4 x 25416 x 1152 10.5 and 8.7). Where most SMs have two and K is long it wins again:
// 8 x 28672 x 4096 21.6 and 22.3, 8 x 8192 x 28672 38.0 and 41.8; one or two rows are less work: 1 x 6144 x 4096 8.8 and 9.1. Over
// 401 sizes of 1..8 rows, in a graph and one by one, this rule gains 4 % where it takes the kernel and is nowhere more than 5 % behind.
// At 16 rows the quantiser warps no longer keep up with the weights at all: four projections of a 4096-wide layer 56.6 and 65.0 us
// (with twice as many of them 56.2, but then 1 row takes 50.3 instead of 48.0).
static bool quant_in_gemm_wins(int64_t M, int64_t N, int64_t K, int sms, int splits) {
  const int64_t ctas = cdiv(N, 128) * splits, kb = cdiv(cdiv(K, 128), splits);
  return ctas <= sms - 16 || (3 * ctas > 4 * sms && kb >= 15) ||
         (M <= 2 && ((ctas > sms && kb >= 15) || (splits > 1 && 9 * ctas > 10 * sms && kb >= 7)));
}
static bool linear_quant_in_gemm(int64_t M, int64_t N, int64_t K, int sms, GemmRoute* route) {
  const Tuning& tune = tuning();
  const bool forced = tune.linear_decode_fused == 2;  // the launch refuses what the kernel cannot take
  if (M > (forced ? kLinearStreamMaxM : SkinnyCfg<16, true>::kQuantRows) || tune.linear_decode_fused == 0 || tune.gemm_splitk > 0 || tune.gemm_bn >= 0) return false;
  const GemmPlan plan = plan_gemm(M, N, K, sms, true);
  const SkinnySplit split = skinny_split(M, N, K, plan.splits);
  if (!plan.skinny || !split.direct()) return false;
  if (!forced && !quant_in_gemm_wins(M, N, K, sms, split.splits)) return false;
  *route = skinny_route(M, N, K, plan.splits, false, B200_KERNEL_SKINNY_QUANT);
  return true;
}
// A linear layer: one of the two kernels that quantise their input themselves, or the quantiser and what route_gemm says.
static GemmRoute route_linear(int64_t M, int64_t N, int64_t K, int sms) {
  GemmRoute r;
  int ranks;
  if (linear_one_launch(M, N, K, sms, &ranks))
    return {B200_KERNEL_STREAM_QUANT, 256, ranks, ranks > 1 ? B200_SUM_CLUSTER : B200_SUM_NONE};
  const int gemm_sms = sms < 148 ? sms : 148;
  if (linear_quant_in_gemm(M, N, K, gemm_sms, &r)) return r;
  return route_gemm(M, N, K, gemm_sms);
}
}  // namespace b200

extern "C" size_t b200_w8a8_block_fp8_linear_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (linear_one_launch(M, N, K, sm_count())) return 0;
  return linear_q_bytes(M, K) + linear_s_bytes(M, K) + b200_w8a8_block_fp8_gemm_workspace_bytes(M, N, K);
}

extern "C" int b200_w8a8_block_fp8_linear(const void* x, int x_dtype, const void* B, const float* Bs, void* out, int64_t M,
                                          int64_t N, int64_t K, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace b200;
  B200_CHECK_ARG(M >= 0 && N >= 0 && K > 0, "linear: bad shape");
  if (M == 0 || N == 0) return B200_OK;
  B200_UNSUPPORTED(x_dtype != B200_BF16 && x_dtype != B200_F16, "linear: 16-bit activations only (dtype code %d)", x_dtype);
  B200_UNSUPPORTED(K % 128 != 0, "linear: K=%lld must be a multiple of 128", (long long)K);
  B200_CHECK_ARG(x && B && Bs && out, "linear: null pointer");
  B200_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)B & 15) == 0, "linear: x and B must be 16-byte aligned");
  B200_UNSUPPORTED(N % 8 != 0, "linear: N=%lld must be a multiple of 8", (long long)N);
  GemmRoute r = {};
  if (M <= kLinearStreamMaxM) r = route_linear(M, N, K, sm_count());  // no kernel takes more rows as they come
  if (r.kernel == B200_KERNEL_STREAM_QUANT) return run_linear_stream(x, x_dtype, B, Bs, out, M, N, K, 1e-10f, static_cast<cudaStream_t>(stream));
  if (r.kernel == B200_KERNEL_SKINNY_QUANT) {
    B200_CHECK_ARG(((uintptr_t)out & 15) == 0, "gemm: A, B and C must be 16-byte aligned");
    B200_UNSUPPORTED(N > 0x7fffff00LL || K > 0x7fffff00LL, "gemm: dimension too large");
    SkinnyParams sp = {};
    sp.x = x; sp.eps = 1e-10f; sp.Bs = Bs;
    return run_skinny(nullptr, B, sp, r, out, x_dtype, M, N, K, nullptr, 0, static_cast<cudaStream_t>(stream), FanOut{});
  }
  const size_t need = b200_w8a8_block_fp8_linear_workspace_bytes(M, N, K);
  if (need && (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255) != 0)) {
    set_error_detail("linear: workspace %zu < %zu bytes or not 256-byte aligned", workspace_bytes, need);
    return B200_E_WORKSPACE;
  }
  uint8_t* q = static_cast<uint8_t*>(workspace);
  float* s = reinterpret_cast<float*>(q + linear_q_bytes(M, K));
  uint8_t* rest = reinterpret_cast<uint8_t*>(s) + linear_s_bytes(M, K);
  int rc = quant_for_linear(x, x_dtype, q, s, M, K, static_cast<cudaStream_t>(stream));
  if (rc) return rc;
  return gemm_impl(q, s, 1, M, B, Bs, out, x_dtype, M, N, K, rest, need - (size_t)(rest - q), stream, FanOut{});
}

extern "C" size_t b200_w8a8_block_fp8_linear_decode_workspace_bytes(int64_t, int64_t, int64_t) { return 0; }

extern "C" int b200_w8a8_block_fp8_linear_decode(const void* x, int x_dtype, const void* B, const float* Bs, void* out,
                                                 int64_t M, int64_t N, int64_t K, float eps, void* workspace,
                                                 size_t workspace_bytes, void* tickets, void* stream) {
  using namespace b200;
  (void)workspace, (void)workspace_bytes;  // the K split is summed through distributed shared memory
  B200_CHECK_ARG(M >= 0 && N >= 0 && K > 0, "linear_decode: bad shape");
  if (M == 0 || N == 0) return B200_OK;
  B200_UNSUPPORTED(M > kLinearStreamMaxM, "linear_decode: M=%lld rows (at most %d)", (long long)M, (int)kLinearStreamMaxM);
  B200_UNSUPPORTED(x_dtype != B200_BF16 && x_dtype != B200_F16, "linear_decode: 16-bit activations only (dtype code %d)", x_dtype);
  B200_UNSUPPORTED(K % 16 != 0 || N % 8 != 0, "linear_decode: K=%lld must be a multiple of 16, N=%lld of 8", (long long)K,
                   (long long)N);
  B200_UNSUPPORTED(N > 4096 * 128, "linear_decode: N=%lld is too large", (long long)N);
  B200_CHECK_ARG(x && B && Bs && out && tickets, "linear_decode: null pointer");
  B200_CHECK_ARG(((uintptr_t)x & 15) == 0 && ((uintptr_t)B & 15) == 0, "linear_decode: x and B must be 16-byte aligned");
  return run_linear_stream(x, x_dtype, B, Bs, out, M, N, K, eps, static_cast<cudaStream_t>(stream));
}

namespace b200 {
// Modelled time of the block-scaled kernels (see plan_gemm; fitted to 590 sizes of 65..2200 rows, within 8 %): launch and set-up, whole
// waves of tiles, a CTA's 128 x 224 at 0.34 us per 128-K block, a pair's 256 x 240 at 0.30, and the operands, of which a pair halves
// what it reads of the weights: 160 x 14336 x 4096 18.8 and 17.8 us, 3000 x 4096 x 14336 2244 and 2759 TFLOP/s; 1500 x 2560 x 4096
// 15.7 and 16.6, 400 x 8192 x 1024 8.1 and 9.8.
static double block_scaled_us(int64_t M, int64_t N, int64_t K, int sms, bool pair) {
  if (pair && sms < 2) return 1e30;
  const double num_kb = (double)cdiv(K, 128), weights = (double)N * (double)K / 1e6, rows = (double)M * (double)K / 1e6;
  if (N < 256) return (pair ? 4.4 : 3.0) + (N > 128 ? 1.0 : 0.0) + num_kb * 0.26;  // narrow, few tiles: 2135 x 80 x 256 3.5 us
  if (pair)
    return 4.73 + (double)cdiv(cdiv(M, 256) * cdiv(N, Ue8m0PairCfg::BN), sms / 2) * (num_kb * 0.303 + 0.99) + 0.019 * weights + 0.051 * rows;
  return 3.46 + (double)cdiv(cdiv(M, 128) * cdiv(N, Ue8m0Cfg::BN), sms) * (num_kb * 0.343 + 0.96) + 0.027 * weights;
}
static bool block_scaled_pair(int64_t M, int64_t N, int64_t K, int sms) {
  const long knob = tuning().gemm_ue8m0;
  return knob == 2 || (knob != 1 && block_scaled_us(M, N, K, sms, true) <= block_scaled_us(M, N, K, sms, false));
}
}  // namespace b200

extern "C" int b200_w8a8_block_fp8_gemm_ue8m0(const void* A, const int32_t* sfa, int64_t sfa_ld, const void* B,
                                              const int32_t* sfb, int64_t sfb_ld, int sfb_rows_per_word, void* C,
                                              int c_dtype, int64_t M, int64_t N, int64_t K, void* stream) {
  using namespace b200;
  B200_CHECK_ARG(M >= 0 && N >= 0 && K > 0, "gemm_ue8m0: bad shape");
  if (M == 0 || N == 0) return B200_OK;
  B200_CHECK_ARG(A && B && C && sfa && sfb, "gemm_ue8m0: null pointer");
  B200_CHECK_ARG(((uintptr_t)A & 15) == 0 && ((uintptr_t)B & 15) == 0 && ((uintptr_t)C & 15) == 0,
                 "gemm_ue8m0: A, B and C must be 16-byte aligned");
  B200_CHECK_ARG(sfb_rows_per_word == 1 || sfb_rows_per_word == 128, "gemm_ue8m0: one scale word per row or per 128 rows of B");
  B200_CHECK_ARG(sfa_ld >= M && sfb_ld >= cdiv(N, sfb_rows_per_word), "gemm_ue8m0: scale row pitch shorter than the rows");
  B200_UNSUPPORTED(K % 16 != 0 || N % 8 != 0, "gemm_ue8m0: K=%lld must be a multiple of 16, N=%lld of 8", (long long)K,
                   (long long)N);
  B200_UNSUPPORTED(M > 0x7fffff00LL || N > 0x7fffff00LL || K > 0x7fffff00LL, "gemm_ue8m0: dimension too large");
  Ue8m0Params p = {};
  p.sfa = sfa; p.sfb = sfb; p.sfa_ld = sfa_ld; p.sfb_ld = sfb_ld; p.sfb_rows_per_word = sfb_rows_per_word;
  p.C = C; p.M = (int)M; p.N = (int)N; p.K = (int)K;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (block_scaled_pair(M, N, K, plan_sms())) {
    switch (c_dtype) {
      case B200_BF16: return launch_gemm_ue8m0_pair<__nv_bfloat16>(A, B, p, st);
      case B200_F16: return launch_gemm_ue8m0_pair<__half>(A, B, p, st);
      case B200_F32: return launch_gemm_ue8m0_pair<float>(A, B, p, st);
      default: break;
    }
  }
  switch (c_dtype) {
    case B200_BF16: return launch_gemm_ue8m0<__nv_bfloat16>(A, B, p, st);
    case B200_F16: return launch_gemm_ue8m0<__half>(A, B, p, st);
    case B200_F32: return launch_gemm_ue8m0<float>(A, B, p, st);
    default:
      set_error_detail("gemm_ue8m0: unknown output dtype code %d", c_dtype);
      return B200_E_BAD_ARG;
  }
}

// ---------------------------------------------------------------- packed power-of-two scales, any M
namespace b200 {
// Packed exponent words -> the fp32 scales of the promotion kernels (exact): As column-major [num_kb][M], Bs
// [n_blocks][num_kb]. One thread per word of four K blocks.
__global__ void __launch_bounds__(256) unpack_scales_kernel(const int32_t* __restrict__ sfa, int64_t sfa_ld,
                                                            const int32_t* __restrict__ sfb, int64_t sfb_ld, int sfb_step,
                                                            float* __restrict__ as, float* __restrict__ bs, int M, int n_blocks,
                                                            int num_kb) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int words = (num_kb + 3) / 4;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < (int64_t)M * words) {
    const int w = (int)(i / M), m = (int)(i - (int64_t)w * M);
    const uint32_t e = (uint32_t)__ldg(sfa + w * sfa_ld + m);
    for (int k = 0; k < 4 && 4 * w + k < num_kb; ++k) as[(int64_t)(4 * w + k) * M + m] = __uint_as_float((e >> (8 * k) & 0xffu) << 23);
  } else if (i - (int64_t)M * words < (int64_t)n_blocks * words) {
    const int j = (int)(i - (int64_t)M * words), w = j / n_blocks, n = j - w * n_blocks;
    const uint32_t e = (uint32_t)__ldg(sfb + w * sfb_ld + (int64_t)n * sfb_step);
    for (int k = 0; k < 4 && 4 * w + k < num_kb; ++k) bs[(int64_t)n * num_kb + 4 * w + k] = __uint_as_float((e >> (8 * k) & 0xffu) << 23);
  }
}

constexpr double kUnpackUs = 1.1;
// Whether the block-scaled kernels (scales applied by the tensor core, no K split) beat the promotion kernels on unpacked
// scales, or the decode kernel, which reads the packed words itself: below 65 rows the weight stream decides, then the modelled
// times (which know nothing of the power cap, at which applying scales in the tensor core pays: 4 %). The choice is 0.6 % behind
// the best on those sizes (203 x 4096 x 14336: 46 us block-scaled, 25 promoted; 96 x 5120 x 1536 9.4 and 7.2 in the decode
// kernel; 204 x 336 x 1152 6.6 and 4.9; 1500 x 4096 x 14336 75.7 and 85.5).
static bool block_scaled_wins(int64_t M, int64_t N, int64_t K, int sms) {
  if (tuning().gemm_ue8m0 > 0) return true;
  if (M <= 64) return false;
  const double one = block_scaled_us(M, N, K, sms, false), two = block_scaled_us(M, N, K, sms, true);
  return (one < two ? one : two) <= plan_gemm(M, N, K, sms, true, PlanFor{false, kUnpackUs}).us * (N < 256 ? 1.0 : 1.04);
}
static size_t packed_as_bytes(int64_t M, int64_t K) { return align_up((size_t)(M * cdiv(K, 128)) * 4, 256); }
static size_t packed_bs_bytes(int64_t N, int64_t K) { return align_up((size_t)(cdiv(N, 128) * cdiv(K, 128)) * 4, 256); }
}  // namespace b200

extern "C" size_t b200_w8a8_block_fp8_gemm_packed_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0 || block_scaled_wins(M, N, K, plan_sms())) return 0;
  // the decode kernel takes its partials first, the others run on unpacked scales with the plain plan
  const size_t partials = partial_bytes(M, N, K), decode = partial_bytes(M, N, K, PlanFor{false, kUnpackUs});
  return packed_as_bytes(M, K) + packed_bs_bytes(N, K) + (partials > decode ? partials : decode);
}

extern "C" int b200_w8a8_block_fp8_gemm_packed(const void* A, const int32_t* sfa, int64_t sfa_ld, const void* B,
                                               const int32_t* sfb, int64_t sfb_ld, int sfb_rows_per_word, void* C, int c_dtype,
                                               int64_t M, int64_t N, int64_t K, void* workspace, size_t workspace_bytes,
                                               void* stream) {
  using namespace b200;
  B200_CHECK_ARG(M >= 0 && N >= 0 && K > 0, "gemm_packed: bad shape");
  if (M == 0 || N == 0) return B200_OK;
  const size_t need = b200_w8a8_block_fp8_gemm_packed_workspace_bytes(M, N, K);
  if (need == 0)
    return b200_w8a8_block_fp8_gemm_ue8m0(A, sfa, sfa_ld, B, sfb, sfb_ld, sfb_rows_per_word, C, c_dtype, M, N, K, stream);
  B200_CHECK_ARG(sfa && sfb, "gemm_packed: null pointer");
  B200_CHECK_ARG(sfb_rows_per_word == 1 || sfb_rows_per_word == 128, "gemm_packed: one scale word per row or per 128 rows of B");
  B200_CHECK_ARG(sfa_ld >= M && sfb_ld >= cdiv(N, sfb_rows_per_word), "gemm_packed: scale row pitch shorter than the rows");
  B200_UNSUPPORTED(M > 0x7fffff00LL || N > 0x7fffff00LL || K > 0x7fffff00LL, "gemm_packed: dimension too large");
  if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255) != 0) {
    set_error_detail("gemm_packed: workspace %zu < %zu bytes or not 256-byte aligned", workspace_bytes, need);
    return B200_E_WORKSPACE;
  }
  const GemmRoute r = route_gemm(M, N, K, plan_sms(), PlanFor{false, kUnpackUs});
  if (r.kernel == B200_KERNEL_SKINNY && tuning().gemm_splitk <= 0) {  // a few rows: the decode kernel reads the packed words itself
    B200_CHECK_ARG(A && B && C && ((uintptr_t)A & 15) == 0 && ((uintptr_t)B & 15) == 0 && ((uintptr_t)C & 15) == 0,
                   "gemm_packed: A, B and C must be 16-byte aligned");
    B200_CHECK_ARG(c_dtype == B200_BF16 || c_dtype == B200_F16 || c_dtype == B200_F32, "gemm_packed: unknown output dtype code %d", c_dtype);
    B200_UNSUPPORTED(K % 16 != 0 || N % 8 != 0, "gemm_packed: K=%lld must be a multiple of 16, N=%lld of 8", (long long)K, (long long)N);
    SkinnyParams sp = {};
    sp.sfa = sfa; sp.sfb = sfb; sp.sfa_ld = sfa_ld; sp.sfb_ld = sfb_ld; sp.sfb_step = 128 / sfb_rows_per_word;
    return run_skinny(A, B, sp, r, C, c_dtype, M, N, K, workspace, workspace_bytes, static_cast<cudaStream_t>(stream), FanOut{});
  }
  float* as = static_cast<float*>(workspace);
  uint8_t* bs = static_cast<uint8_t*>(workspace) + packed_as_bytes(M, K);
  uint8_t* rest = bs + packed_bs_bytes(N, K);
  const int n_blocks = (int)cdiv(N, 128), num_kb = (int)cdiv(K, 128);
  const int64_t total = (M + n_blocks) * cdiv(num_kb, 4);
  int rc = launch_dependent(unpack_scales_kernel, dim3((unsigned)cdiv(total, 256)), 256, 0, static_cast<cudaStream_t>(stream), 1,
                            "unpack_scales_kernel", sfa, sfa_ld, sfb, sfb_ld, 128 / sfb_rows_per_word, as,
                            reinterpret_cast<float*>(bs), (int)M, n_blocks, num_kb);
  if (rc) return rc;
  return gemm_impl(A, as, 1, M, B, reinterpret_cast<const float*>(bs), C, c_dtype, M, N, K, rest,
                   need - (size_t)(rest - static_cast<uint8_t*>(workspace)), stream, FanOut{});
}

extern "C" int b200_plan_dense(int entry, int64_t M, int64_t N, int64_t K, int sms, int* kernel, int* tile_n, int* splits, int* sum) {
  using namespace b200;
  B200_CHECK_ARG(entry >= B200_PLAN_GEMM && entry <= B200_PLAN_GEMM_PACKED, "plan: unknown entry point code %d", entry);
  B200_CHECK_ARG(M > 0 && N > 0 && K > 0 && sms >= 0, "plan: bad shape");
  B200_CHECK_ARG(kernel && tile_n && splits && sum, "plan: null pointer");
  if (sms == 0) sms = sm_count();
  const int gemm_sms = sms < 148 ? sms : 148;
  GemmRoute r;
  if (entry == B200_PLAN_LINEAR)
    r = route_linear(M, N, K, sms);
  else if (entry == B200_PLAN_GEMM_PACKED && block_scaled_wins(M, N, K, gemm_sms))
    r = block_scaled_pair(M, N, K, gemm_sms) ? GemmRoute{B200_KERNEL_BLOCK_SCALED_PAIR, Ue8m0PairCfg::BN, 1, B200_SUM_NONE}
                                             : GemmRoute{B200_KERNEL_BLOCK_SCALED, Ue8m0Cfg::BN, 1, B200_SUM_NONE};
  else
    r = route_gemm(M, N, K, gemm_sms, PlanFor{entry == B200_PLAN_GEMM_FANOUT, entry == B200_PLAN_GEMM_PACKED ? kUnpackUs : 0.0});
  *kernel = r.kernel, *tile_n = r.tile_n, *splits = r.splits, *sum = r.sum;
  return B200_OK;
}
