// fused_experts(use_fp8_w8a8=True, block_shape=[128,128]) for sm_100a.
//
// Launch sequence (all on the caller's stream, no host sync):
//   1 align            token->expert buckets padded to 16 .. 128 rows           (align.cu)
//   2 scatter_quant    hidden rows -> expert-sorted FP8 rows + 1x128 scales     (HBM bound)
//     (up to 1024 pairs of the weight-streaming path: 1 and 2 in one launch)
//   3 grouped GEMM 1   sorted rows x w1[expert]^T; the epilogue applies silu(gate)*up in fp32
//                      and re-quantises to FP8 + 1x128 scales from the accumulators (tcgen05)
//   4 grouped GEMM 2   x w2[expert]^T, * router weight, scattered to (token, slot)
//   5 sum_reduce       fp32 sum over the top-k slots -> out                     (HBM bound)
// Scales of the two intermediate activations are stored column-major ([K/128][rows]) so a
// GEMM promotion warp reads 32 consecutive floats per K block.
#include <math.h>
#include <stdlib.h>

#include "gemm_host.cuh"
#include "gemm_stream.cuh"

namespace b200 {

constexpr int kMoeBlockM = 128;

// Token rows -> expert-sorted FP8 rows + scales: one block per token quantises (or reads) its row once and writes it to
// the positions of all of its pairs, so a 16-bit row is read once instead of once per pair (or quantised, written and
// read back). Blocks past the tokens zero pad rows. HBM-bound by the sorted rows written: 16384 tokens of 7168 to 8 experts
// each, quantiser + gather 465 us, this kernel 250.
// 8 consecutive lanes share a 128-group; a thread holds 16 consecutive elements.
constexpr int kPadSlots = 32;     // sorted slots a pad block looks at
constexpr int kRowScales = 1024;  // groups of a row whose scales are written together
template <typename T>
__global__ void __launch_bounds__(512) moe_scatter_quant_kernel(
    const T* __restrict__ hidden, const uint8_t* __restrict__ hidden_q, const float* __restrict__ hidden_s,
    const int32_t* __restrict__ position, const int32_t* __restrict__ sorted_ids, const int32_t* __restrict__ num_post_pad,
    uint8_t* __restrict__ q, float* __restrict__ s, int64_t T_tokens, int64_t H, int numel, int topk, int64_t s_row, int64_t s_group) {
  if (blockIdx.x >= T_tokens) {
    // Pad rows: a GEMM output row depends on its own A row only and rows computed from pad slots are never scattered,
    // so their content is free. Zeros keep the tensor cores' power draw down when tiles are mostly real rows; with a few
    // tokens per expert writing them would dominate this kernel, and the launch leaves these blocks out.
    const int64_t slot0 = ((int64_t)blockIdx.x - T_tokens) * kPadSlots;
    // every warp looks at the slots at once (kPadSlots == 32) and then only at the pads among them
    const int64_t slot = slot0 + (threadIdx.x & 31);
    unsigned pads = __ballot_sync(0xffffffffu, slot < *num_post_pad && __ldg(sorted_ids + slot) >= numel);
    for (; pads; pads &= pads - 1) {
      const int r = __ffs(pads) - 1;
      for (int chunk = threadIdx.x; chunk < H / 16; chunk += blockDim.x) {
        *reinterpret_cast<uint4*>(q + (slot0 + r) * H + chunk * 16) = make_uint4(0, 0, 0, 0);
        if ((chunk & 7) == 0) s[(slot0 + r) * s_row + (chunk / 8) * s_group] = 0.f;
      }
    }
    return;
  }
  __shared__ int pos[64];
  __shared__ float row_s[kRowScales];
  const int64_t tok = blockIdx.x;
  for (int j = threadIdx.x; j < min(topk, 64); j += blockDim.x) pos[j] = __ldg(position + tok * topk + j);
  __syncthreads();
  // more than 64 slots per token: the scatter entry point takes them (fused_experts and the slot sum refuse)
  auto position_of = [&](int j) { return j < 64 ? pos[j] : __ldg(position + tok * topk + j); };
  const int groups = (int)(H / 128);
  for (int c0 = threadIdx.x & ~31; c0 < H / 16; c0 += blockDim.x) {  // whole warps
    const int chunk = c0 + (threadIdx.x & 31);
    const bool active = chunk < H / 16;
    uint4 out;
    float scale;
    if (hidden_q != nullptr) {
      out = active ? ld_nc_16(hidden_q + tok * H + chunk * 16) : make_uint4(0, 0, 0, 0);
      scale = active && (chunk & 7) == 0 ? __ldg(hidden_s + tok * (H / 128) + chunk / 8) : 0.f;
    } else {
      uint4 raw[2];
      raw[0] = active ? ld_nc_16(hidden + tok * H + chunk * 16) : make_uint4(0, 0, 0, 0);
      raw[1] = active ? ld_nc_16(hidden + tok * H + chunk * 16 + 8) : make_uint4(0, 0, 0, 0);
      scale = quant_chunk<T>(raw, 1e-10f, out);
    }
    if (!active) continue;
    if ((chunk & 7) == 0 && chunk / 8 < kRowScales) row_s[chunk / 8] = scale;
    for (int j = 0; j < topk; ++j) {
      const int64_t p = position_of(j);
      if (p < 0) continue;  // an expert on another rank
      *reinterpret_cast<uint4*>(q + p * H + chunk * 16) = out;
      if ((chunk & 7) == 0 && chunk / 8 >= kRowScales) s[p * s_row + (chunk / 8) * s_group] = scale;
    }
  }
  __syncthreads();
  const int kept = min(groups, kRowScales);
  for (int i = threadIdx.x; i < topk * kept; i += blockDim.x) {  // consecutive threads -> consecutive groups of one row
    const int j = i / kept, g = i - j * kept;
    const int64_t p = position_of(j);
    if (p >= 0) s[p * s_row + g * s_group] = row_s[g];
  }
}

// A few pairs (the weight-streaming path): align, quantise and gather in ONE launch, one block per (token, slot)
// pair. The position of a pair in the expert-sorted layout is the padded size of the lower experts' runs plus its
// rank among the pairs of its expert: two sums over a histogram and one over the ids, cheap enough for every block
// to redo (numel <= 1024) instead of passing them through memory between three kernels. Same layout as
// moe_align_block_size, without the runs of ids that are not on this rank. One token of 256 experts: 3 kernels, 9.5 us
// plus two launch gaps -> one of 5 us.
constexpr int kPrepMaxPairs = 1024;
template <typename T>
__global__ void __launch_bounds__(256) moe_prep_kernel(const T* __restrict__ hidden, const uint8_t* __restrict__ hidden_q,
                                                       const float* __restrict__ hidden_s, const int32_t* __restrict__ topk_ids,
                                                       int32_t* __restrict__ sorted, int32_t* __restrict__ expert_ids,
                                                       int32_t* __restrict__ npp, uint8_t* __restrict__ q,
                                                       float* __restrict__ s, int64_t H, int E, int numel, int topk, int block_m,
                                                       int64_t cap) {
  __shared__ int cnt[1024];
  __shared__ int part[3][8];
  const int tid = threadIdx.x, i = blockIdx.x;
  for (int b = tid; b < E; b += 256) cnt[b] = 0;
  grid_dependency_wait();
  grid_launch_dependents();
  __syncthreads();
  const int mine = __ldg(topk_ids + i);
  const bool valid = mine >= 0 && mine < E;
  if (!valid && i != 0) return;
  int rank = 0;
  for (int j = tid; j < numel; j += 256) {
    const int e = __ldg(topk_ids + j);
    if (e >= 0 && e < E) {
      atomicAdd(&cnt[e], 1);
      rank += (e == mine && j < i) ? 1 : 0;
    }
  }
  __syncthreads();
  int before = 0, total = 0;
  for (int b = tid; b < E; b += 256) {
    const int padded = (cnt[b] + block_m - 1) / block_m * block_m;
    total += padded;
    before += b < mine ? padded : 0;
  }
  rank = __reduce_add_sync(0xffffffffu, rank);
  before = __reduce_add_sync(0xffffffffu, before);
  total = __reduce_add_sync(0xffffffffu, total);
  if ((tid & 31) == 0) part[0][tid >> 5] = rank, part[1][tid >> 5] = before, part[2][tid >> 5] = total;
  __syncthreads();
  rank = before = total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) rank += part[0][w], before += part[1][w], total += part[2][w];
  if (i == 0 && tid == 0) *npp = total;
  if (!valid) return;
  const int pos = before + rank, run = cnt[mine];
  if (tid == 0) {
    sorted[pos] = i;
    if (rank % block_m == 0) expert_ids[pos / block_m] = mine;
  }
  if (rank == run - 1)  // the last pair of an expert marks the pad rows behind it
    for (int k = run + tid; k < (run + block_m - 1) / block_m * block_m; k += 256) sorted[before + k] = numel;
  const int64_t tok = i / topk;
  for (int c0 = tid & ~31; c0 < H / 16; c0 += 256) {  // whole warps; 8 consecutive lanes share a 128-group
    const int chunk = c0 + (tid & 31);
    const bool active = chunk < H / 16;
    uint4 out;
    float scale;
    if (hidden_q != nullptr) {
      out = active ? ld_nc_16(hidden_q + tok * H + chunk * 16) : make_uint4(0, 0, 0, 0);
      scale = active && (chunk & 7) == 0 ? __ldg(hidden_s + tok * (H / 128) + chunk / 8) : 0.f;
    } else {
      uint4 raw[2];
      raw[0] = active ? ld_nc_16(hidden + tok * H + chunk * 16) : make_uint4(0, 0, 0, 0);
      raw[1] = active ? ld_nc_16(hidden + tok * H + chunk * 16 + 8) : make_uint4(0, 0, 0, 0);
      scale = quant_chunk<T>(raw, 1e-10f, out);
    }
    if (!active) continue;
    *reinterpret_cast<uint4*>(q + (int64_t)pos * H + chunk * 16) = out;
    if ((chunk & 7) == 0) s[(int64_t)(chunk / 8) * cap + pos] = scale;
  }
}

// out[t, :] = scale * sum_j y[t*topk + j, :] over the slots whose expert id is valid. One block per token: the
// valid slots are listed once in shared memory, so a row none of whose slots is valid (most rows of an
// expert-parallel receive area) costs one read of its ids, and there is no per-thread division. Four row loads
// are in flight per thread and six blocks fit an SM; the sum stays in slot order.
constexpr int kSumReduceMaxSlots = 64;
template <typename T>
__global__ void __launch_bounds__(256, 6) moe_sum_reduce_kernel(const T* __restrict__ y, const int32_t* __restrict__ topk_ids,
                                                                T* __restrict__ out, int topk, int E, int64_t H, float scale,
                                                                int skip_unrouted, const int* __restrict__ poison_status) {
  __shared__ int s_slot[kSumReduceMaxSlots];
  __shared__ int s_n;
  const int64_t t = blockIdx.x;
  grid_launch_dependents();
  grid_dependency_wait();
  if (poison_status != nullptr && *reinterpret_cast<const volatile int*>(poison_status) != 0) {
    // the rows were to be written by other GPUs and the handshake before this kernel gave up: NaNs, not stale rows
    const uint4 nan16 = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);  // NaN in bf16 and fp16
    for (int64_t c = (blockIdx.y * blockDim.x + threadIdx.x) * 8; c < H; c += (int64_t)gridDim.y * blockDim.x * 8) *reinterpret_cast<uint4*>(out + t * H + c) = nan16;
    return;
  }
  if (threadIdx.x < 32) {  // warp 0 compacts the valid slots, ascending (topk <= 64: two rounds of 32)
    int n = 0;
    for (int j0 = 0; j0 < topk; j0 += 32) {
      const int j = j0 + (int)threadIdx.x;
      const int e = j < topk ? __ldg(topk_ids + t * topk + j) : -1;
      const bool ok = e >= 0 && e < E;
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (ok) s_slot[n + __popc(m & ((1u << threadIdx.x) - 1u))] = j;
      n += __popc(m);
    }
    if (threadIdx.x == 0) s_n = n;
  }
  __syncthreads();
  const int n = s_n;
  if (n == 0 && skip_unrouted) return;  // a row no local expert serves: nobody reads it
  const int vec_per_row = (int)(H / 8);
  const T* base = y + t * topk * H;
  for (int v = blockIdx.y * blockDim.x + threadIdx.x; v < vec_per_row; v += gridDim.y * blockDim.x) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int k0 = 0; k0 < n; k0 += 4) {
      uint4 r[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k0 + k < n) r[k] = ld_nc_16(base + (int64_t)s_slot[k0 + k] * H + v * 8);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k0 + k < n) {
          const T* h = reinterpret_cast<const T*>(&r[k]);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] += to_f32<T>(h[i]);
        }
      }
    }
    uint4 o;
    T* oh = reinterpret_cast<T*>(&o);
#pragma unroll
    for (int i = 0; i < 8; ++i) oh[i] = from_f32<T>(acc[i] * scale);
    *reinterpret_cast<uint4*>(out + t * H + v * 8) = o;
  }
}

// Same reduction over fp32 split-K partials y[splits][rows * slots][H] of the down GEMM
// (few-token case): out[r, :] = scale * sum over valid slots j and splits s. Rows whose slots
// are all invalid come out as zeros.
template <typename T>
__global__ void __launch_bounds__(256) moe_sum_reduce_splits_kernel(const float* __restrict__ y,
                                                                    const int32_t* __restrict__ topk_ids,
                                                                    T* __restrict__ out, int64_t rows, int slots,
                                                                    int splits, int64_t split_stride, int E, int64_t H,
                                                                    float scale, int skip_unrouted) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int vec_per_row = (int)(H / 8);
  if (c >= rows * vec_per_row) return;
  const int64_t r = c / vec_per_row;
  const int v = (int)(c - r * vec_per_row);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  bool any = false;
  for (int j = 0; j < slots; ++j) {
    const int e = topk_ids[r * slots + j];
    if (e < 0 || e >= E) continue;
    any = true;
    for (int sp = 0; sp < splits; ++sp) {
      const float* src = y + sp * split_stride + (r * slots + j) * H + v * 8;
      const uint4 a = ld_nc_16(src), b = ld_nc_16(src + 4);
      acc[0] += __uint_as_float(a.x); acc[1] += __uint_as_float(a.y);
      acc[2] += __uint_as_float(a.z); acc[3] += __uint_as_float(a.w);
      acc[4] += __uint_as_float(b.x); acc[5] += __uint_as_float(b.y);
      acc[6] += __uint_as_float(b.z); acc[7] += __uint_as_float(b.w);
    }
  }
  if (!any && skip_unrouted) return;
  uint4 o;
  T* oh = reinterpret_cast<T*>(&o);
#pragma unroll
  for (int i = 0; i < 8; ++i) oh[i] = from_f32<T>(acc[i] * scale);
  *reinterpret_cast<uint4*>(out + r * H + v * 8) = o;
}

// Split-K factor of the down GEMM. With a handful of tokens the live tiles (about one 128-row
// tile per routed expert, H/256 column tiles each) leave most SMs without weights to stream;
// K = I is then split and the fp32 partials are summed by the slot reduction.
static int moe_down_k_splits(int64_t numel, int E, int64_t H, int64_t I, int sms) {
  const int64_t live = (numel < E ? numel : E) + numel / kMoeBlockM;
  const int64_t tiles = live * cdiv(H, 256);
  const int64_t num_kb = I / 128;
  if (tiles * 4 >= (int64_t)sms * 3 || num_kb < 8) return 1;
  int64_t s = sms / tiles;
  if (s > num_kb / 4) s = num_kb / 4;
  if (s > 8) s = 8;
  return s < 2 ? 1 : (int)s;
}

struct MoeWorkspace {
  int block_m;  // rows per expert block of the sorted layout
  int64_t cap;  // rows of the expert-sorted layout (multiple of block_m)
  int64_t cap_blocks;
  int down_splits;  // > 1: the down GEMM writes fp32 split-K partials instead of 16-bit rows
  size_t off_sorted, off_expert, off_npp, off_cumsum, off_align, off_aq1, off_as1, off_aq2, off_as2, off_c3, off_pos, total;
};

// Rows per expert block of the sorted layout, and with it the kernel: 16 / 32 / 64 for the weight-streaming kernel,
// 128 for the tile kernel. An expert's weights are read once per block of its rows, so the block should hold the
// rows of a busy expert; a wider one only adds columns of padding. With evenly loaded experts a busy one has about
// avg + 2 sqrt(avg) rows; with few experts the router skews more and the hottest ones set the time: twice the
// average. Layer times in us for blocks of 16 / 32 / 64 / 128 rows: 256 experts (7168 x 2048) at 8 rows on average
// 1807 / 1795 / 1944 / 2202, 16: 2178 / 1825 / 1958 / 2169, 32: 2854 / 2160 / 1968 / 2172, 64: 4044 / 2978 / 2736 /
// 2257; 8 skewed experts (4096 x 14336) at 4: 207 / 216 / 237 / 240, 8: 269 / 241 / 266 / 270, 32: 422 / 346 / 356 / 292.
static int moe_block_rows(int64_t numel, int E) {
  const long knob = tuning().moe_decode;
  if (knob == 0) return kMoeBlockM;
  if (knob == 16 || knob == 32 || knob == 64) return (int)knob;
  const double avg = (double)numel / (double)(numel < E ? numel : E);
  const double busy = (E <= 32 ? 2.0 : 1.0) * avg + 2.0 * sqrt(avg);
  if (busy <= 16) return 16;
  if (busy <= 32) return 32;
  if (busy <= 64 || knob == 1) return 64;
  return kMoeBlockM;
}

static MoeWorkspace moe_workspace_layout(int64_t T, int topk, int E, int64_t H, int64_t I, bool tile_only) {
  MoeWorkspace w = {};
  const int64_t numel = T * topk;
  w.block_m = tile_only ? kMoeBlockM : moe_block_rows(numel, E);
  const int64_t max_pad = numel < E + 1 ? numel * w.block_m : numel + (int64_t)(E + 1) * (w.block_m - 1);
  w.cap = cdiv(max_pad, w.block_m) * w.block_m;
  w.cap_blocks = w.cap / w.block_m;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o = align_up(o + bytes, 256); return at; };
  w.off_sorted = take((size_t)w.cap * 4);
  w.off_expert = take((size_t)w.cap_blocks * 4);
  w.off_npp = take(4);
  w.off_cumsum = take((size_t)(E + 2) * 4);
  w.off_align = take(b200_moe_align_workspace_bytes(numel, E + 1));
  w.off_aq1 = take((size_t)w.cap * H);
  w.off_as1 = take((size_t)w.cap * (H / 128) * 4);
  w.off_aq2 = take((size_t)w.cap * I);
  w.off_as2 = take((size_t)w.cap * (I / 128) * 4);
  w.down_splits = moe_down_k_splits(numel, E, H, I, sm_count());
  w.off_c3 = take(w.down_splits > 1 ? (size_t)w.down_splits * numel * H * 4 : (size_t)numel * H * 2);
  w.off_pos = take((size_t)numel * 4);
  w.total = o;
  return w;
}

// The two grouped GEMMs over token blocks of NT rows (see gemm_stream.cuh).
template <int NT, typename T>
static int run_stream_gemms(const uint8_t* aq1, const float* as1, uint8_t* aq2, float* as2, const void* w1, const void* w2,
                            const float* w1_scale, const float* w2_scale, const float* topk_weights, int weight_on_input,
                            T* rows, int E, int64_t H, int64_t I, int64_t cap, StreamParams p, cudaStream_t st) {
  p.as_ld = cap;
  p.As = as1; p.Bs = w1_scale; p.n_out = (int)I; p.q_out = aq2; p.q_scales = as2; p.q_ld = cap;
  p.topk_weights = weight_on_input ? topk_weights : nullptr;
  int rc = launch_stream<NT, STREAM_GATE_UP, T>(w1, (int64_t)E * 2 * I, aq1, cap, H, p, st);
  if (rc) return rc;
  p.As = as2; p.Bs = w2_scale; p.n_out = (int)H; p.C = rows;
  p.topk_weights = weight_on_input ? nullptr : topk_weights;
  return launch_stream<NT, STREAM_DOWN, T>(w2, (int64_t)E * H, aq2, cap, I, p, st);
}

// Destinations of the (token, slot) rows when they leave for several buffers (expert-parallel combine by push).
struct ScatterDests {
  void* dest[8];
  int n;
  int64_t rows_per_dest;
};

template <typename T>
static int run_fused_experts(const void* hidden, const float* hidden_scale, const void* w1, const void* w2, const float* w1_scale,
                             const float* w2_scale, const float* topk_weights, const int32_t* topk_ids, void* out,
                             int64_t T_tokens, int topk, int E, int64_t H, int64_t I, int combine_mode,
                             int weight_on_input, float routed_scale, uint8_t* ws, cudaStream_t st,
                             const ScatterDests* scatter = nullptr) {
  if (scatter != nullptr) combine_mode = B200_COMBINE_NONE;  // rows leave per (token, slot); the receiver sums
  const int no_combine = combine_mode == B200_COMBINE_NONE;
  const int skip_unrouted = combine_mode == B200_COMBINE_SUM_SKIP_UNROUTED;
  // rows that leave for several buffers are sent by the tile kernel's epilogue
  const MoeWorkspace L = moe_workspace_layout(T_tokens, topk, E, H, I, scatter != nullptr);
  const int64_t numel = T_tokens * topk;
  int32_t* sorted = reinterpret_cast<int32_t*>(ws + L.off_sorted);
  int32_t* expert_ids = reinterpret_cast<int32_t*>(ws + L.off_expert);
  int32_t* npp = reinterpret_cast<int32_t*>(ws + L.off_npp);
  int32_t* cumsum = reinterpret_cast<int32_t*>(ws + L.off_cumsum);
  uint8_t* aq1 = ws + L.off_aq1;
  float* as1 = reinterpret_cast<float*>(ws + L.off_as1);
  uint8_t* aq2 = ws + L.off_aq2;
  float* as2 = reinterpret_cast<float*>(ws + L.off_as2);
  int down_splits = L.down_splits;
  if (tuning().moe_down_splitk == 0) down_splits = 1;  // knob: keep the 16-bit single-pass path
  const bool stream = L.block_m != kMoeBlockM;
  // Layout of the sorted rows' scales: [H/128][cap] is what the GEMMs read fastest (a warp's 32 rows are one run), but
  // with several pairs per token the scatter then writes many single floats (16384 tokens to 8 experts: 70 us)
  const bool scales_by_row = !stream && topk >= 4;
  if (scatter != nullptr || stream) down_splits = 1;   // rows go straight to their receivers in 16 bits
  const bool split = down_splits > 1;
  T* c3 = no_combine && !split ? static_cast<T*>(out) : reinterpret_cast<T*>(ws + L.off_c3);

  int rc = B200_OK;
  const bool one_launch = stream && numel <= kPrepMaxPairs && E <= 1024;
  if (!one_launch) {
    rc = align_with_inverse(topk_ids, numel, E + 1, L.block_m, sorted, L.cap, expert_ids, L.cap_blocks, npp, cumsum,
                            reinterpret_cast<int32_t*>(ws + L.off_pos), ws + L.off_align, st);
    if (rc) return rc;
  }
  if (no_combine && !split && scatter == nullptr) {
    // rows of slots whose expert is not on this rank are never written by GEMM 2
    cudaError_t e = cudaMemsetAsync(out, 0, (size_t)numel * H * sizeof(T), st);
    if (e != cudaSuccess) {
      set_error_detail("memset(out): %s", cudaGetErrorString(e));
      return B200_E_LAUNCH;
    }
  }
  if (one_launch) {
    rc = launch_dependent(moe_prep_kernel<T>, dim3((unsigned)numel), 256, 0, st, 1, "moe_prep_kernel",
                          hidden_scale ? nullptr : static_cast<const T*>(hidden),
                          hidden_scale ? static_cast<const uint8_t*>(hidden) : nullptr, hidden_scale, topk_ids, sorted,
                          expert_ids, npp, aq1, as1, H, E, (int)numel, topk, L.block_m, L.cap);
    if (rc) return rc;
  } else {
    // zero pad rows where on average a quarter of a tile per expert or more is real
    bool zero_pads = numel >= (int64_t)E * 32;
    if (tuning().moe_zero_pads >= 0) zero_pads = tuning().moe_zero_pads != 0;
    const int64_t blocks = T_tokens + (zero_pads ? cdiv(L.cap, kPadSlots) : 0);
    const int threads = H / 16 < 512 ? (int)cdiv(H / 16, 32) * 32 : 512;
    moe_scatter_quant_kernel<T><<<(unsigned)blocks, threads, 0, st>>>(
        hidden_scale ? nullptr : static_cast<const T*>(hidden), hidden_scale ? static_cast<const uint8_t*>(hidden) : nullptr,
        hidden_scale, reinterpret_cast<const int32_t*>(ws + L.off_pos), sorted, npp, aq1, as1, T_tokens, H, (int)numel, topk,
        scales_by_row ? H / 128 : 1, scales_by_row ? 1 : L.cap);
    if ((rc = check_launch("moe_scatter_quant_kernel"))) return rc;
  }
  if (stream) {
    StreamParams sp = {};
    sp.expert_ids = expert_ids; sp.num_post_pad = npp; sp.sorted_ids = sorted; sp.numel = (int)numel; sp.experts = E;
    // Every bucket that has rows has at most one partly filled block. The separate align lays out the pairs of other ranks
    // (id -1) as a bucket of its own, in front of the experts'; moe_prep_kernel leaves them out.
    const int64_t buckets = one_launch ? E : E + 1;
    const int64_t bound = (numel < buckets ? numel : buckets) + numel / L.block_m;
    sp.max_blocks = (int)(bound < L.cap_blocks ? bound : L.cap_blocks);
#define B200_STREAM(NT)                                                                                                    \
  run_stream_gemms<NT, T>(aq1, as1, aq2, as2, w1, w2, w1_scale, w2_scale, topk_weights, weight_on_input, c3, E, H, I, \
                          L.cap, sp, st)
    rc = L.block_m == 16 ? B200_STREAM(16) : L.block_m == 32 ? B200_STREAM(32) : B200_STREAM(64);
#undef B200_STREAM
    if (rc) return rc;
    if (no_combine) return B200_OK;
    // a few tokens: several blocks per token, one 16-byte vector per thread
    const unsigned cols = T_tokens <= 512 ? (unsigned)cdiv(H / 8, 256) : 1u;
    return launch_dependent(moe_sum_reduce_kernel<T>, dim3((unsigned)T_tokens, cols), 256, 0, st, 1, "moe_sum_reduce", c3,
                            topk_ids, static_cast<T*>(out), topk, E, H, routed_scale, skip_unrouted, nullptr);
  }
  const int force_bn = tuning().gemm_bn == 128 || tuning().gemm_bn == 256 ? (int)tuning().gemm_bn : 0;
  GemmParams p = {};
  p.expert_ids = expert_ids; p.num_post_pad = npp; p.sorted_ids = sorted; p.numel = (int)numel;
  p.M = (int)L.cap;
  // GEMM 1: [cap, H] x w1[E, 2I, H]^T -> silu(gate)*up -> FP8 [cap, I] + column-major scales
  p.As = as1; p.as_sm = scales_by_row ? H / 128 : 1; p.as_sk = scales_by_row ? 1 : L.cap; p.Bs = w1_scale; p.C = nullptr; p.ldc = 0;
  p.N = (int)I; p.K = (int)H; p.topk_weights = weight_on_input ? topk_weights : nullptr;
  p.q_out = aq2; p.q_scales = as2; p.q_scale_ld = L.cap;
  if ((rc = launch_gemm<GEMM_GROUPED_SILU_QUANT, T>(aq1, w1, (int64_t)E * 2 * I, p, 256, st))) return rc;
  // GEMM 2: [cap, I] x w2[E, H, I]^T -> rows scattered to (token, slot), times the router weight
  p.As = as2; p.as_sm = 1; p.as_sk = L.cap; p.Bs = w2_scale; p.C = c3; p.ldc = H; p.N = (int)H; p.K = (int)I;
  p.topk_weights = weight_on_input ? nullptr : topk_weights;
  if (scatter != nullptr) {
    p.C = nullptr;
    p.scatter_rows_per_dest = (int)scatter->rows_per_dest;
    p.scatter_div = make_fastdiv((int)scatter->rows_per_dest);
    for (int d = 0; d < scatter->n; ++d) p.dest[d] = scatter->dest[d];
  }
  if (split) {
    p.split_stride = numel * H;
    if ((rc = launch_gemm<GEMM_GROUPED_SCATTER, float>(aq2, w2, (int64_t)E * H, p, 256, st, down_splits)))
      return rc;
    const int64_t rows = no_combine ? numel : T_tokens;
    const int64_t total = rows * (H / 8);
    moe_sum_reduce_splits_kernel<T><<<(unsigned)cdiv(total, 256), 256, 0, st>>>(
        reinterpret_cast<const float*>(c3), topk_ids, static_cast<T*>(out), rows, no_combine ? 1 : topk, down_splits,
        numel * H, E, H, no_combine ? 1.0f : routed_scale, skip_unrouted);
    return check_launch("moe_sum_reduce_splits");
  }
  if ((rc = launch_gemm<GEMM_GROUPED_SCATTER, T>(aq2, w2, (int64_t)E * H, p, force_bn, st))) return rc;
  if (!no_combine) {
    moe_sum_reduce_kernel<T><<<(unsigned)T_tokens, 256, 0, st>>>(c3, topk_ids, static_cast<T*>(out), topk, E, H,
                                                                  routed_scale, skip_unrouted, nullptr);
    if ((rc = check_launch("moe_sum_reduce"))) return rc;
  }
  return B200_OK;
}

// ---------------------------------------------------------------- masked (low-latency) layout
// Tokens arrive already grouped by expert: hidden [E][T_pad][H] with the first masked_m[e] rows of
// expert e valid (what a low-latency expert-parallel dispatch delivers). The grouped GEMMs above
// run unchanged on that layout: row tile mt belongs to expert mt / (T_pad/128) and is skipped
// when it starts at or beyond masked_m[e]; rows past masked_m[e] inside a live tile are computed
// and dropped by the store predicate (their "destination" is the out-of-range index).
__global__ void __launch_bounds__(256) masked_meta_kernel(const int32_t* __restrict__ masked_m, int32_t* __restrict__ sorted,
                                                          int32_t* __restrict__ expert_ids, int32_t* __restrict__ npp,
                                                          int E, int64_t T_pad) {
  const int64_t cap = (int64_t)E * T_pad;
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (row == 0) *npp = (int32_t)cap;
  if (row >= cap) return;
  const int e = (int)(row / T_pad);
  const int64_t r = row - (int64_t)e * T_pad;
  const int m = min(max(masked_m[e], 0), (int)T_pad);
  sorted[row] = r < m ? (int32_t)row : (int32_t)cap;
  if (r % kMoeBlockM == 0) expert_ids[row / kMoeBlockM] = r < m ? e : -1;
}

struct MaskedWorkspace {
  int64_t cap;
  size_t off_sorted, off_expert, off_npp, off_aq2, off_as2, total;
};

static MaskedWorkspace masked_workspace_layout(int E, int64_t T_pad, int64_t I) {
  MaskedWorkspace w = {};
  w.cap = (int64_t)E * T_pad;
  size_t o = 0;
  auto take = [&](size_t bytes) { size_t at = o; o = align_up(o + bytes, 256); return at; };
  w.off_sorted = take((size_t)w.cap * 4);
  w.off_expert = take((size_t)(w.cap / kMoeBlockM) * 4);
  w.off_npp = take(4);
  w.off_aq2 = take((size_t)w.cap * I);
  w.off_as2 = take((size_t)w.cap * (I / 128) * 4);
  w.total = o;
  return w;
}

template <typename T>
static int run_masked_experts(const void* hidden_q, const float* hidden_s, const void* w1, const void* w2,
                              const float* w1_scale, const float* w2_scale, const int32_t* masked_m, void* out, int E,
                              int64_t T_pad, int64_t H, int64_t I, uint8_t* ws, cudaStream_t st) {
  const MaskedWorkspace L = masked_workspace_layout(E, T_pad, I);
  int32_t* sorted = reinterpret_cast<int32_t*>(ws + L.off_sorted);
  int32_t* expert_ids = reinterpret_cast<int32_t*>(ws + L.off_expert);
  int32_t* npp = reinterpret_cast<int32_t*>(ws + L.off_npp);
  uint8_t* aq2 = ws + L.off_aq2;
  float* as2 = reinterpret_cast<float*>(ws + L.off_as2);
  masked_meta_kernel<<<(unsigned)cdiv(L.cap, 256), 256, 0, st>>>(masked_m, sorted, expert_ids, npp, E, T_pad);
  int rc = check_launch("masked_meta_kernel");
  if (rc) return rc;
  GemmParams p = {};
  p.expert_ids = expert_ids; p.num_post_pad = npp; p.sorted_ids = sorted; p.numel = (int)L.cap;
  p.M = (int)L.cap;
  // gate_up: row-major input scales [cap][H/128]
  p.As = hidden_s; p.as_sm = H / 128; p.as_sk = 1; p.Bs = w1_scale; p.N = (int)I; p.K = (int)H;
  p.q_out = aq2; p.q_scales = as2; p.q_scale_ld = L.cap;
  if ((rc = launch_gemm<GEMM_GROUPED_SILU_QUANT, T>(hidden_q, w1, (int64_t)E * 2 * I, p, 256, st))) return rc;
  // down: rows stay where they are (identity "scatter"), no router weight
  p.As = as2; p.as_sm = 1; p.as_sk = L.cap; p.Bs = w2_scale; p.C = out; p.ldc = H; p.N = (int)H; p.K = (int)I;
  return launch_gemm<GEMM_GROUPED_SCATTER, T>(aq2, w2, (int64_t)E * H, p, 0, st);
}

}  // namespace b200

extern "C" size_t b200_masked_experts_fp8_workspace_bytes(int E, int64_t T_pad, int64_t H, int64_t I) {
  if (E <= 0 || T_pad <= 0 || H <= 0 || I <= 0) return 0;
  return b200::masked_workspace_layout(E, T_pad, I).total;
}

extern "C" int b200_masked_experts_fp8(const void* hidden_q, const float* hidden_s, const void* w1, const void* w2,
                                       const float* w1_scale, const float* w2_scale, const int32_t* masked_m, void* out,
                                       int out_dtype, int E, int64_t T_pad, int64_t H, int64_t I, void* workspace,
                                       size_t workspace_bytes, void* stream) {
  using namespace b200;
  B200_CHECK_ARG(E > 0 && T_pad > 0 && H > 0 && I > 0, "masked_experts: bad shape");
  B200_CHECK_ARG(hidden_q && hidden_s && w1 && w2 && w1_scale && w2_scale && masked_m && out, "masked_experts: null pointer");
  B200_UNSUPPORTED(T_pad % 128 != 0, "masked_experts: T_pad=%lld must be a multiple of 128", (long long)T_pad);
  B200_UNSUPPORTED(H % 128 != 0 || I % 128 != 0, "masked_experts: H=%lld and I=%lld must be multiples of 128",
                   (long long)H, (long long)I);
  B200_UNSUPPORTED((int64_t)E * T_pad >= (1LL << 30), "masked_experts: too many rows");
  B200_CHECK_ARG(((uintptr_t)hidden_q & 15) == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)w1 & 15) == 0 &&
                     ((uintptr_t)w2 & 15) == 0, "masked_experts: tensors must be 16-byte aligned");
  const size_t need = b200_masked_experts_fp8_workspace_bytes(E, T_pad, H, I);
  if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255) != 0) {
    set_error_detail("masked_experts: workspace %zu < %zu bytes or not 256-byte aligned", workspace_bytes, need);
    return B200_E_WORKSPACE;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  if (out_dtype == B200_BF16)
    return run_masked_experts<__nv_bfloat16>(hidden_q, hidden_s, w1, w2, w1_scale, w2_scale, masked_m, out, E, T_pad, H, I, ws, st);
  if (out_dtype == B200_F16)
    return run_masked_experts<__half>(hidden_q, hidden_s, w1, w2, w1_scale, w2_scale, masked_m, out, E, T_pad, H, I, ws, st);
  set_error_detail("masked_experts: output dtype code %d is not bf16/f16", out_dtype);
  return B200_E_UNSUPPORTED;
}

extern "C" size_t b200_fused_experts_fp8_workspace_bytes(int64_t T, int topk, int E, int64_t H, int64_t I) {
  if (T <= 0 || topk <= 0 || E <= 0 || H <= 0 || I <= 0) return 0;
  // the layout with 128-row blocks is the larger one, and either may be used with this size
  return b200::moe_workspace_layout(T, topk, E, H, I, true).total;
}

extern "C" int b200_fused_experts_fp8(const void* hidden, const float* hidden_scale, int h_dtype, const void* w1,
                                      const void* w2,
                                      const float* w1_scale, const float* w2_scale, const float* topk_weights,
                                      const int32_t* topk_ids, void* out, int64_t T, int topk, int E, int64_t H,
                                      int64_t I, int no_combine, int apply_router_weight_on_input,
                                      float routed_scaling_factor, void* workspace, size_t workspace_bytes,
                                      void* stream) {
  using namespace b200;
  B200_CHECK_ARG(T >= 0 && topk > 0 && E > 0 && H > 0 && I > 0, "fused_experts: bad shape");
  if (T == 0) return B200_OK;
  B200_CHECK_ARG(hidden && w1 && w2 && w1_scale && w2_scale && topk_weights && topk_ids && out,
                 "fused_experts: null pointer");
  B200_UNSUPPORTED(H % 128 != 0 || I % 128 != 0, "fused_experts: H=%lld and I=%lld must be multiples of 128",
                   (long long)H, (long long)I);
  B200_UNSUPPORTED(E + 1 > 1025, "fused_experts: more than 1024 experts");
  B200_UNSUPPORTED(T * topk >= (1LL << 30), "fused_experts: too many (token, slot) pairs");
  B200_UNSUPPORTED(topk > kSumReduceMaxSlots, "fused_experts: more than %d experts per token", kSumReduceMaxSlots);
  B200_CHECK_ARG(!apply_router_weight_on_input || topk == 1, "apply_router_weight_on_input needs topk == 1");
  B200_CHECK_ARG(no_combine >= 0 && no_combine <= 2, "fused_experts: unknown combine mode %d", no_combine);
  B200_CHECK_ARG(((uintptr_t)hidden & 15) == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)w1 & 15) == 0 &&
                     ((uintptr_t)w2 & 15) == 0, "fused_experts: tensors must be 16-byte aligned");
  const size_t need = b200_fused_experts_fp8_workspace_bytes(T, topk, E, H, I);
  if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255) != 0) {
    set_error_detail("fused_experts: workspace %zu < %zu bytes or not 256-byte aligned", workspace_bytes, need);
    return B200_E_WORKSPACE;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  if (h_dtype == B200_BF16)
    return run_fused_experts<__nv_bfloat16>(hidden, hidden_scale, w1, w2, w1_scale, w2_scale, topk_weights, topk_ids, out, T, topk, E,
                                            H, I, no_combine, apply_router_weight_on_input, routed_scaling_factor, ws, st);
  if (h_dtype == B200_F16)
    return run_fused_experts<__half>(hidden, hidden_scale, w1, w2, w1_scale, w2_scale, topk_weights, topk_ids, out, T, topk, E, H, I,
                                     no_combine, apply_router_weight_on_input, routed_scaling_factor, ws, st);
  set_error_detail("fused_experts: hidden dtype code %d is not bf16/f16", h_dtype);
  return B200_E_UNSUPPORTED;
}

extern "C" int b200_fused_experts_fp8_scatter(const void* hidden_q, const float* hidden_scale, int out_dtype, const void* w1,
                                              const void* w2, const float* w1_scale, const float* w2_scale,
                                              const float* topk_weights, const int32_t* topk_ids, void* const* dests,
                                              int n_dest, int64_t rows_per_dest, int64_t T, int topk, int E, int64_t H,
                                              int64_t I, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace b200;
  B200_CHECK_ARG(T >= 0 && topk > 0 && E > 0 && H > 0 && I > 0, "fused_experts_scatter: bad shape");
  if (T == 0) return B200_OK;
  B200_CHECK_ARG(hidden_q && hidden_scale && w1 && w2 && w1_scale && w2_scale && topk_weights && topk_ids && dests,
                 "fused_experts_scatter: null pointer (rows arrive quantised: FP8 bytes + scales)");
  B200_CHECK_ARG(n_dest >= 1 && n_dest <= 8 && rows_per_dest > 0 && rows_per_dest < (1LL << 30) &&
                     (int64_t)n_dest * rows_per_dest >= T * topk,
                 "fused_experts_scatter: %d destinations x %lld rows do not cover %lld pairs", n_dest,
                 (long long)rows_per_dest, (long long)(T * topk));
  B200_UNSUPPORTED(H % 128 != 0 || I % 128 != 0, "fused_experts_scatter: H=%lld and I=%lld must be multiples of 128",
                   (long long)H, (long long)I);
  B200_UNSUPPORTED(E + 1 > 1025, "fused_experts_scatter: more than 1024 experts");
  B200_UNSUPPORTED(T * topk >= (1LL << 30), "fused_experts_scatter: too many (token, slot) pairs");
  ScatterDests sd = {};
  sd.n = n_dest;
  sd.rows_per_dest = rows_per_dest;
  for (int d = 0; d < n_dest; ++d) {
    B200_CHECK_ARG(dests[d] && ((uintptr_t)dests[d] & 15) == 0, "fused_experts_scatter: destination %d null or unaligned", d);
    sd.dest[d] = dests[d];
  }
  B200_CHECK_ARG(((uintptr_t)hidden_q & 15) == 0 && ((uintptr_t)w1 & 15) == 0 && ((uintptr_t)w2 & 15) == 0,
                 "fused_experts_scatter: tensors must be 16-byte aligned");
  const size_t need = b200_fused_experts_fp8_workspace_bytes(T, topk, E, H, I);
  if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255) != 0) {
    set_error_detail("fused_experts_scatter: workspace %zu < %zu bytes or not 256-byte aligned", workspace_bytes, need);
    return B200_E_WORKSPACE;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  if (out_dtype == B200_BF16)
    return run_fused_experts<__nv_bfloat16>(hidden_q, hidden_scale, w1, w2, w1_scale, w2_scale, topk_weights, topk_ids, nullptr, T,
                                            topk, E, H, I, B200_COMBINE_NONE, 0, 1.0f, ws, st, &sd);
  if (out_dtype == B200_F16)
    return run_fused_experts<__half>(hidden_q, hidden_scale, w1, w2, w1_scale, w2_scale, topk_weights, topk_ids, nullptr, T, topk,
                                     E, H, I, B200_COMBINE_NONE, 0, 1.0f, ws, st, &sd);
  set_error_detail("fused_experts_scatter: output dtype code %d is not bf16/f16", out_dtype);
  return B200_E_UNSUPPORTED;
}

extern "C" int b200_moe_sum_reduce(const void* rows, const int32_t* topk_ids, void* out, int dtype, int64_t T, int topk, int E,
                                   int64_t H, float scale, int skip_unrouted, int poison_on_status, void* stream) {
  using namespace b200;
  B200_CHECK_ARG(T >= 0 && topk > 0 && E > 0 && H > 0 && H % 8 == 0, "moe_sum_reduce: bad shape");
  if (T == 0) return B200_OK;
  B200_CHECK_ARG(rows && topk_ids && out && ((uintptr_t)rows & 15) == 0 && ((uintptr_t)out & 15) == 0,
                 "moe_sum_reduce: null or unaligned pointer");
  B200_UNSUPPORTED(topk > kSumReduceMaxSlots, "moe_sum_reduce: more than %d experts per token", kSumReduceMaxSlots);
  B200_UNSUPPORTED(T >= (1LL << 31), "moe_sum_reduce: too many tokens");
  const int* status = poison_on_status ? device_status_word() : nullptr;
  if (poison_on_status && !status) {
    set_error_detail("cannot resolve the device status word");
    return B200_E_LAUNCH;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == B200_BF16)
    moe_sum_reduce_kernel<__nv_bfloat16><<<(unsigned)T, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(rows), topk_ids,
                                                                       static_cast<__nv_bfloat16*>(out), topk, E, H, scale,
                                                                       skip_unrouted, status);
  else if (dtype == B200_F16)
    moe_sum_reduce_kernel<__half><<<(unsigned)T, 256, 0, st>>>(static_cast<const __half*>(rows), topk_ids,
                                                                static_cast<__half*>(out), topk, E, H, scale, skip_unrouted, status);
  else {
    set_error_detail("moe_sum_reduce: dtype code %d is not bf16/f16", dtype);
    return B200_E_UNSUPPORTED;
  }
  return check_launch("moe_sum_reduce");
}
