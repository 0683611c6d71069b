// Shared device/host helpers for the mixlab_b200 kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <utility>

#include "../../include/mixlab_b200.h"

namespace mxb {

// Numeric guards of the reference's chunked scan (gpu/ir.cpp:35-37).
constexpr float kGateFloor = 1e-30f;
constexpr float kLogGateFloor = -69.07755278982137f;  // log(1e-30)
constexpr float kExpClampMin = -80.0f;

// exp(clamp(x, -80, 0)) - stable_exp_nonpos, gpu/ir.cpp:903-905.
__device__ __forceinline__ float exp_nonpos(float x) {
  return __expf(fminf(fmaxf(x, kExpClampMin), 0.0f));
}
// Full-precision variant for the fp32 parity path.
__device__ __forceinline__ float exp_nonpos_precise(float x) {
  return expf(fminf(fmaxf(x, kExpClampMin), 0.0f));
}

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <typename F>
__device__ __forceinline__ F warp_sum(F v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of 8 columns over the 32 lanes of a warp: v[c] is this lane's value for column c.  Recursive halving, 9 shuffles
// instead of 40.  On return lane l holds in v[0] the sum of column l & 7.
template <int M, int N>
__device__ __forceinline__ void colsum8_step(float (&v)[8], int lane) {
  const bool up = (lane & M) != 0;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float send = up ? v[k] : v[k + N];
    const float keep = up ? v[k + N] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, M);
  }
}
__device__ __forceinline__ void colsum8(float (&v)[8], int lane) {
  colsum8_step<4, 4>(v, lane);
  colsum8_step<2, 2>(v, lane);
  colsum8_step<1, 1>(v, lane);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 8);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// Reverse inclusive cumulative sum over 64 values by one warp, two per lane: call with a = x[63 - 2 lane],
// b = x[62 - 2 lane]; returns in a, b the sums x[63] + ... + x[63 - 2 lane] and ... + x[62 - 2 lane].  A fixed order.
template <typename F>
__device__ __forceinline__ void warp_rcumsum64(F& a, F& b, int lane) {
  F v = a + b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const F t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  a = v - b;
  b = v;
}

// Sums over `rows` rows of 16 (TALL) or 32 columns in a fixed order; part: the calling thread's column, put(c, sum) is called once
// for each column c of the CTA.  TALL: 1024 threads, 64 slices of them take every 64th row, the slices are added pairwise across a
// warp and then by a warp per column; otherwise 256 threads and 8 slices.  Eight loads in flight a thread.  Few columns want the
// first (1184 rows of 448 columns 17.7 us with 8 slices, 3.8 with 64: it is the latency of the loads), columns enough to fill the
// GPU the second (256 rows of 12,320 columns 6.0 with 8, 12.3 with 64): col_sum_tall().
template <bool TALL>
constexpr int kSumCols = TALL ? 16 : 32;
template <bool TALL>
constexpr int kSumThreads = TALL ? 1024 : 256;
inline bool col_sum_tall(size_t columns) { return columns <= 16 * 2 * 148; }
template <bool TALL, typename F>
__device__ __forceinline__ void col_sum(const float* __restrict__ part, size_t rows, size_t pitch, bool in, F&& put) {
  constexpr int COLS = kSumCols<TALL>, SLICES = kSumThreads<TALL> / COLS;
  __shared__ float red[32][COLS + 1];
  const int col = threadIdx.x % COLS, slice = threadIdx.x / COLS, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float s = 0.f;
  if (in) {
    const float* src = part + slice * pitch;
    const size_t step = SLICES * pitch;
    int left = ((int)rows - slice + SLICES - 1) / SLICES;
    for (; left >= 8; left -= 8, src += 8 * step) {
      float v[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) v[x] = __ldg(src + x * step);
#pragma unroll
      for (int x = 0; x < 8; ++x) s += v[x];
    }
    float v[7];
#pragma unroll
    for (int x = 0; x < 7; ++x) v[x] = x < left ? __ldg(src + x * step) : 0.f;
#pragma unroll
    for (int x = 0; x < 7; ++x) s += v[x];
  }
  if (TALL) s += __shfl_xor_sync(0xffffffffu, s, COLS & 31);  // two slices a warp
  if (lane < COLS) red[warp][col] = s;
  __syncthreads();
  if constexpr (TALL) {
    const float t = warp_sum(warp < COLS ? red[lane][warp] : 0.f);
    if (lane == 0 && warp < COLS) put(warp, t);
  } else if (warp == 0) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < SLICES; ++k) t += red[k][lane];
    put(lane, t);
  }
}

// First statement of a kernel that launch_kernel() starts: nothing is read or written before the kernels in front of it in the
// stream are done and their writes visible.
__device__ __forceinline__ void begin_dependent() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- host side ----------------------------------------------------------
// Launch that is prepared while the kernel in front of it in the stream still runs (programmatic dependent launch): its blocks
// take their places as soon as the last blocks in front have left, without waiting for their writes to drain and for the
// launch itself.  Every kernel started so begins with begin_dependent().  No kernel gives its permission earlier
// (griddepcontrol.launch_dependents): the blocks behind it would crowd on the SMs that are free first.  us a call, plain
// launches / this / with the permission at the start of every kernel: float32 forward 2 x 256 x 4 heads 26.9 / 22.5 / 28.7,
// Mamba-3 float32 2 x 1024 x 128 channels (12 launches) 111 / 87 / 95, Mamba-3 1 x 200 x 8 heads 62 / 50 / 49, gated delta
// rule on float32 tensors 4 x 2048 x 16 heads 461 / 443 / 470.  These are calls back to back, the boundary between two calls
// included (with a copy of the inputs in front of each call, 3.1 us, the float32 forward: 29.7 / 24.6); a caller that waits for
// each call gains at the launches within it only.
template <typename... P, typename... A>
inline void launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);  // (a failure is what check_launch reads)
}
void note_launch(int n = 1);           // bumps mxb_launch_count()
mxb_status check_launch(const char* what);  // cudaGetLastError -> status
void set_last_cuda_error(int e);
// Optional per-launch CUDA-event tracing (mxb_trace_enable); no-ops when off.
void trace_begin(const char* name, cudaStream_t st);
void trace_end(cudaStream_t st);

// Launch wrapper: counts the launch and, when tracing is on, brackets it with events.
#define MXB_LAUNCH(name, st, ...)   \
  do {                              \
    ::mxb::trace_begin(name, st);   \
    __VA_ARGS__;                    \
    ::mxb::trace_end(st);           \
    ::mxb::note_launch();           \
  } while (0)

// Opts a kernel in to more than 48 KB of dynamic shared memory, once per device and kernel (the attribute belongs to the
// device's context): done is the caller's record, one bit per device.
mxb_status allow_smem(const void* kernel, int bytes, std::atomic<uint64_t>& done);
#define MXB_ALLOW_SMEM(bytes, ...)                                              \
  ([&]() -> mxb_status {                                                        \
    static std::atomic<uint64_t> done{0};                                       \
    return ::mxb::allow_smem(reinterpret_cast<const void*>(__VA_ARGS__), bytes, done); \
  }())

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Carves a caller-provided workspace into 256-byte aligned pieces.
struct Carver {
  char* base;
  size_t off = 0;
  explicit Carver(void* p) : base(static_cast<char*>(p)) {}
  template <typename T>
  T* take(size_t count) {
    off = align_up(off, 256);
    T* r = base ? reinterpret_cast<T*>(base + off) : nullptr;
    off += count * sizeof(T);
    return r;
  }
  size_t bytes() const { return align_up(off, 256); }
};

}  // namespace mxb
