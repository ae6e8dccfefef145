// Shared helpers for the sm_100a block-FP8 kernels: status codes, error detail,
// the per-device status word and small device utilities.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../include/b200_blockfp8.h"

namespace b200 {

// Thread-local text describing the last failed call (read by b200_last_error_detail).
void set_error_detail(const char* fmt, ...);

// Address of this device's status word (a __device__ int in status.cu); nullptr on failure.
int* device_status_word();

#define B200_CHECK_ARG(cond, ...)                 \
  do {                                            \
    if (!(cond)) {                                \
      ::b200::set_error_detail(__VA_ARGS__);      \
      return B200_E_BAD_ARG;                      \
    }                                             \
  } while (0)

#define B200_UNSUPPORTED(cond, ...)               \
  do {                                            \
    if (cond) {                                   \
      ::b200::set_error_detail(__VA_ARGS__);      \
      return B200_E_UNSUPPORTED;                  \
    }                                             \
  } while (0)

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error_detail("%s: %s", what, cudaGetErrorString(e));
    return B200_E_LAUNCH;
  }
  return B200_OK;
}

// Process-wide knobs set through b200_set_tuning (tests force a kernel path, tuning sweeps try a
// setting); -1 = decide automatically. Product calls read this struct, never the environment.
struct Tuning {
  long gemm_bn = -1;            // 128 / 256: tile width of the dense GEMM
  long gemm_stream = -1;        // 0 / 1: never / always the dense weight-streaming kernel
  long gemm_skinny = -1;        // 0: never use the decode (swapped-operand) kernel
  long gemm_skinny_max_m = -1;  // rows up to which the decode kernel is used
  long gemm_splitk = -1;        // > 0: forced K split
  long gemm_2cta = -1;          // 0: never the 16-warp kernel, 1 / 2: always, on pairs / single CTAs; 128, 192, 256: pairs of that width;
                                // 1282, 1284: pairs, 128 wide, 2 or 4 K splits summed in clusters
  long gemm_ue8m0 = -1;          // 0: packed power-of-two scales never take the block-scaled MMA kernel
  long linear_decode_fused = -1; // 0: quantiser + GEMM as separate launches at decode sizes, 2: quantiser in the decode GEMM wherever it runs
  long moe_decode = -1;         // 0 / 1: never / always the weight-streaming experts; 16, 32, 64: with that row block
  long moe_down_splitk = -1;    // 0: the down GEMM never splits K
  long moe_zero_pads = -1;      // 0 / 1: whether the gather pass zeroes pad rows
  long peer_wait_ms = -1;       // limit of a device-side wait for another GPU
};
Tuning& tuning();

// Limit of a device-side wait for another GPU (handshakes of the peer-memory collectives), in
// nanoseconds: 2 s unless the peer_wait_ms knob says otherwise (clamped to 100 ms .. 60 s). Ranks
// that can drift further apart than this on the host must synchronise on the host first.
inline unsigned long long peer_wait_ns() {
  long ms = tuning().peer_wait_ms > 0 ? tuning().peer_wait_ms : 2000;
  if (ms < 100) ms = 100;
  if (ms > 60000) ms = 60000;
  return (unsigned long long)ms * 1000000ull;
}


// Launch as a programmatic dependent of the kernel before it in the stream: the grid may be set up while that kernel
// drains. The kernel executes griddepcontrol.wait before it touches global memory that an earlier kernel may use.
// cluster > 1: thread-block clusters of that many blocks along x.
template <typename... P, typename... A>
inline int launch_dependent(void (*k)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, unsigned cluster,
                            const char* what, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, k, P(args)...);
  if (e != cudaSuccess) {
    set_error_detail("%s: %s", what, cudaGetErrorString(e));
    return B200_E_LAUNCH;
  }
  return check_launch(what);
}
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Quantiser of a linear layer (quant.cu): 16-bit x [M, K] -> FP8 rows + column-major scales, launched so that it overlaps
// the kernels on either side.
int quant_for_linear(const void* x, int x_dtype, void* q, float* s, int64_t M, int64_t K, cudaStream_t st);

// moe_align_block_size of int32 ids (align.cu) that also writes every id's position in the sorted layout, -1 for ids that
// are not in [0, num_buckets - 1). ws: b200_moe_align_workspace_bytes.
int align_with_inverse(const int32_t* ids, int64_t numel, int num_buckets, int block_size, int32_t* sorted, int64_t max_pad,
                       int32_t* expert_ids, int64_t max_blocks, int32_t* num_post_pad, int32_t* cumsum, int32_t* inverse,
                       void* ws, cudaStream_t st);

inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// ---------------------------------------------------------------- device utilities
template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// Division by a divisor fixed at launch as a multiply-high and a shift (exact for 0 <= n < 2^31): the 32-bit
// integer division of the hardware is a ~25-instruction dependent chain, and three of them in a row sat on the
// critical path between two tiles of the promotion warps.
struct FastDiv {
  uint32_t mul, shr;
};
inline FastDiv make_fastdiv(int d) {
  FastDiv f = {0u, 0u};
  if (d <= 1) return f;  // mul == 0 marks "divide by one"
  int l = 0;
  while ((1ll << l) < d) ++l;  // ceil(log2 d)
  const int p = 31 + l;
  f.mul = (uint32_t)(((1ull << p) + (uint64_t)d - 1) / (uint64_t)d);
  f.shr = (uint32_t)(p - 32);
  return f;
}
__device__ __forceinline__ int fast_div(int n, FastDiv f) {
  return f.mul == 0u ? n : (int)(__umulhi((uint32_t)n, f.mul) >> f.shr);
}

// 16-byte read-only global load (bypasses L1 allocation: streamed once).
__device__ __forceinline__ uint4 ld_nc_16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// The first n 128-byte K blocks of a weight row into L2. Nothing is read, so a kernel launched as a programmatic dependent
// may ask for its weights while an earlier kernel still writes them: the write goes to the same L2 line.
// Depth, in K blocks per CTA of the dense kernels: what fits the gap before the wait ends; requests beyond that hold up the
// loads behind them. Four projections (6144..28672 x 4096..14336) in a graph, 1 / 16 / 61 rows: none 52.9 / 55.9 / 73.0 us,
// 1 block 51.9 / 55.2 / 73.0, 3 blocks 50.9 / 54.3 / 73.0, 5 blocks 50.2 / 54.3 / 73.7; a rank of eight (10240 x 8192 and so
// on), 61 rows: 1 block 48.9, 3 blocks 49.9, 5 blocks 50.6. Boxes by cp.async.bulk.prefetch.tensor gain nothing, they queue
// in front of the loads. Loads into the ring before the wait, which nothing would order behind a writer: 51.1 / 53.5 / 70.7.
constexpr int kPrefetchKb = 3;
__device__ __forceinline__ void prefetch_weight_row(const uint8_t* row, int n) {
  for (int i = 0; i < n; ++i) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + i * 128) : "memory");
}

// Four consecutive floats from shared memory, read at this point of the program (never cached in
// registers across a barrier wait): for tables another warp fills while this one waits on an mbarrier.
__device__ __forceinline__ float4 ld_shared_f4(const float* p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p)))
               : "memory");
  return v;
}

// Four floats -> four E4M3 bytes (round-to-nearest-even, saturate to +-448), packed little-endian.
__device__ __forceinline__ uint32_t pack4_e4m3(float a, float b, float c, float d) {
  __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return (uint32_t)lo | ((uint32_t)hi << 16);
}

// Unpack 16 elements of type T held in 16-byte registers into fp32.
template <typename T>
struct Vec16;
template <>
struct Vec16<__nv_bfloat16> {
  static constexpr int kLoads = 2;  // 16-byte loads per 16 elements
  __device__ static void load(const __nv_bfloat16* p, float (&f)[16]) {
    uint4 r[2] = {ld_nc_16(p), ld_nc_16(p + 8)};
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(r);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float2 t = __bfloat1622float2(h[i]);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
};
template <>
struct Vec16<__half> {
  __device__ static void load(const __half* p, float (&f)[16]) {
    uint4 r[2] = {ld_nc_16(p), ld_nc_16(p + 8)};
    const __half2* h = reinterpret_cast<const __half2*>(r);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float2 t = __half22float2(h[i]);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
};
template <>
struct Vec16<float> {
  __device__ static void load(const float* p, float (&f)[16]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 r = ld_nc_16(p + 4 * i);
      f[4 * i] = __uint_as_float(r.x);
      f[4 * i + 1] = __uint_as_float(r.y);
      f[4 * i + 2] = __uint_as_float(r.z);
      f[4 * i + 3] = __uint_as_float(r.w);
    }
  }
};

// Quantise 16 fp32 values that share `amax` (already reduced over the group and floored at
// eps) into 16 E4M3 bytes; returns the stored scale. `formula` as in the C ABI.
__device__ __forceinline__ float quant16(const float (&f)[16], float amax, int formula, uint4& out) {
  float s, q[16];
  if (formula == B200_QUANT_V2) {
    s = amax * (1.0f / 448.0f);
    float r = __fdiv_rn(448.0f, amax);
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = f[i] * r;
  } else if (formula == B200_QUANT_RECIP) {
    s = __fdiv_rn(amax, 448.0f);
    float r = __fdiv_rn(1.0f, s);
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = f[i] * r;
  } else if (formula == B200_QUANT_DIV_CORRECTED) {
    s = __fdiv_rn(amax, 448.0f);
    const float r = __frcp_rn(s);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float q0 = f[i] * r;
      // one residual step towards the rounded quotient; a zero result takes the sign of x as x / s does
      q[i] = copysignf(fmaf(fmaf(-q0, s, f[i]), r, q0), f[i]);
    }
  } else {
    s = __fdiv_rn(amax, 448.0f);
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = __fdiv_rn(f[i], s);
  }
  // no explicit clamp to +-448: the conversion below saturates finite values to the same result
  out.x = pack4_e4m3(q[0], q[1], q[2], q[3]);
  out.y = pack4_e4m3(q[4], q[5], q[6], q[7]);
  out.z = pack4_e4m3(q[8], q[9], q[10], q[11]);
  out.w = pack4_e4m3(q[12], q[13], q[14], q[15]);
  return s;
}

// max over the LPG (power of two <= 32) consecutive lanes that share one group.
template <int LPG>
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = LPG / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// 16 consecutive 16-bit elements of a 128-group that 8 consecutive lanes share: bytes and scale as the stand-alone
// quantiser gives them. All 8 lanes call.
template <typename T>
__device__ __forceinline__ float quant_chunk(const uint4 (&raw)[2], float eps, uint4& out) {
  const T* v = reinterpret_cast<const T*>(raw);
  float f[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] = to_f32<T>(v[i]);
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(f[i]));
  amax = fmaxf(group_max<8>(amax), eps);
  return quant16(f, amax, B200_QUANT_DIV_CORRECTED, out);
}

}  // namespace b200
