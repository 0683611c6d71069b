// Element-wise stages of mixlab's canonical Mamba-3 block around the scan
// (mamba3_canonical_block_impl, gpu/ir.cpp:2034-2105):
//   conv  x_branch = causal depthwise conv of x_proj, weight [D, K], tap k multiplies x[t-k]   (:1397-1425)
//   bc    b = RMSNorm(b_proj rows of N, b_norm_scale, eps) + b_bias, same for c                 (:2089-2094)
//   post  out = RMSNorm(y rows of D, post_norm, eps) z sigmoid(z)                               (:2099-2102)
// and their backward passes: HBM streams in 16-byte pieces.  A thread owns 8 consecutive channels (the convolution of float32
// tensors: 4).  Sums over (batch, step) - the weight, scale and bias gradients - go through per-CTA partial rows in the
// workspace and a fixed-order second pass (no atomics).
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace mxb {
namespace m3b {

using bf16 = __nv_bfloat16;
constexpr int kRun = 16;     // steps per lane for the convolution: a whole number of these
constexpr int kMaxK = 4;     // taps

struct BlkP {
  int B, T, D, N, G, K;
  float eps;
  int runs;   // convolution: a lane's steps / kRun
  int wvec;   // convolution: the four taps of a channel can be read at once
};

// C consecutive channels: 8 or 4.
template <typename IO, int C>
__device__ __forceinline__ void load_n(const IO* p, float (&e)[C]) {
  if constexpr (sizeof(IO) == 4) {
#pragma unroll
    for (int i = 0; i < C / 4; ++i) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(p) + i);
      e[4 * i] = a.x; e[4 * i + 1] = a.y; e[4 * i + 2] = a.z; e[4 * i + 3] = a.w;
    }
  } else {
    using V = std::conditional_t<C == 8, uint4, uint2>;
    const V v = __ldg(reinterpret_cast<const V*>(p));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < C / 2; ++i) { e[2 * i] = __low2float(h[i]); e[2 * i + 1] = __high2float(h[i]); }
  }
}
template <typename IO, int C>
__device__ __forceinline__ void store_n(IO* p, const float (&e)[C]) {
  if constexpr (sizeof(IO) == 4) {
#pragma unroll
    for (int i = 0; i < C / 4; ++i)
      reinterpret_cast<float4*>(p)[i] = make_float4(e[4 * i], e[4 * i + 1], e[4 * i + 2], e[4 * i + 3]);
  } else {
    using V = std::conditional_t<C == 8, uint4, uint2>;
    V v;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < C / 2; ++i) h[i] = __floats2bfloat162_rn(e[2 * i], e[2 * i + 1]);
    *reinterpret_cast<V*>(p) = v;
  }
}
template <typename IO>
__device__ __forceinline__ void load8(const IO* p, float (&e)[8]) { load_n<IO, 8>(p, e); }
template <typename IO>
__device__ __forceinline__ void store8(IO* p, const float (&e)[8]) { store_n<IO, 8>(p, e); }
__device__ __forceinline__ float sigmoid_f(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }

// ------------------------------------------------------------------ depthwise convolution
// grid (ceil(D/C / 128), ceil(T / (runs kRun)), B) x 128: thread = C channels (16 bytes of a row, so that the lanes of a warp read
// whole lines), runs kRun steps; weights w[d][k], k < K <= 4.  Loads in flight bound small calls: 4096 x 448 float32 channels,
// forward / backward 12.8 / 13.9 us with eight channels a thread (two loads of 16 bytes, 32 apart; 56 threads of a CTA at work), 8.3
// / 11.7 with four.  In large ones the weights did: 32 loads a thread, each of 32 lines, for 19 of x (8 x 4096 x 2048 bf16, forward
// / backward with the column sums 114 / 203 us); read tap by tap only where they must be, and for up to 64 steps: 65 / 187.  The
// backward takes four channels of bf16 too, so that six CTAs fit an SM (16 bytes spilled): 95.  Of float32 four CTAs of 128 registers
// (96 bytes spilled); with the 241 that it would take, 8 x 4096 x 2048 165 -> 137 us, but 8 x 1024 x 256 8.0 -> 9.1 and 30000 x 5 x 8
// 85 -> 179.
template <typename IO>
constexpr int kConvC = 16 / sizeof(IO);
constexpr int kConvBwdC = 4;  // (the backward's weights, their gradients and six rows of eight channels do not fit a thread's registers)
template <int C>
__device__ __forceinline__ void conv_weights(float (&wk)[kMaxK][C], const float* __restrict__ w, const BlkP& p, int ch) {
  if (p.wvec) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const float4 x = __ldg(reinterpret_cast<const float4*>(w) + ch + c);
      wk[0][c] = x.x; wk[1][c] = x.y; wk[2][c] = x.z; wk[3][c] = x.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kMaxK; ++k)
#pragma unroll
      for (int c = 0; c < C; ++c) wk[k][c] = k < p.K ? w[(size_t)(ch + c) * p.K + k] : 0.f;
  }
}
template <typename IO>
__global__ void __launch_bounds__(128) m3b_conv_fwd_kernel(BlkP p, const IO* __restrict__ x, const float* __restrict__ w,
                                                           IO* __restrict__ y) {
  begin_dependent();
  constexpr int C = kConvC<IO>;
  const int cg = blockIdx.x * 128 + threadIdx.x, ch = cg * C;
  if (ch >= p.D) return;
  const int first = blockIdx.y * p.runs * kRun, b = blockIdx.z;
  float wk[kMaxK][C];
  conv_weights<C>(wk, w, p, ch);
  const IO* __restrict__ xb = x + (size_t)b * p.T * p.D + ch;
  IO* __restrict__ yb = y + (size_t)b * p.T * p.D + ch;
  float x1[C], x2[C], x3[C];
#pragma unroll
  for (int c = 0; c < C; ++c) x1[c] = x2[c] = x3[c] = 0.f;
  if (first - 1 >= 0) load_n<IO, C>(xb + (size_t)(first - 1) * p.D, x1);
  if (first - 2 >= 0) load_n<IO, C>(xb + (size_t)(first - 2) * p.D, x2);
  if (first - 3 >= 0) load_n<IO, C>(xb + (size_t)(first - 3) * p.D, x3);
  for (int t0 = first; t0 < min(p.T, first + p.runs * kRun); t0 += kRun) {
#pragma unroll
    for (int r = 0; r < kRun; ++r) {
      const int t = t0 + r;
      const bool in = t < p.T;
      float x0[C], o[C];
      load_n<IO, C>(xb + (size_t)(in ? t : t0) * p.D, x0);  // clamped address: the loads of the run can all be in flight
#pragma unroll
      for (int c = 0; c < C; ++c) o[c] = wk[0][c] * x0[c] + wk[1][c] * x1[c] + wk[2][c] * x2[c] + wk[3][c] * x3[c];
      if (in) store_n<IO, C>(yb + (size_t)t * p.D, o);
#pragma unroll
      for (int c = 0; c < C; ++c) { x3[c] = x2[c]; x2[c] = x1[c]; x1[c] = x0[c]; }
    }
  }
}
// dx[t] = sum_k w[k] dy[t+k];  dw[d][k] partial = sum over this lane's steps of x[t-k] dy[t]  -> dwp[(b, lane of steps)][k][D]
template <typename IO>
__global__ void __launch_bounds__(128, sizeof(IO) == 2 ? 6 : 4) m3b_conv_bwd_kernel(BlkP p, const IO* __restrict__ x, const float* __restrict__ w,
                                                           const IO* __restrict__ dy, IO* __restrict__ dx,
                                                           float* __restrict__ dwp) {
  begin_dependent();
  constexpr int C = kConvBwdC;
  const int cg = blockIdx.x * 128 + threadIdx.x, ch = cg * C;
  if (ch >= p.D) return;
  const int first = blockIdx.y * p.runs * kRun, b = blockIdx.z;
  float wk[kMaxK][C], dw[kMaxK][C];
  conv_weights<C>(wk, w, p, ch);
#pragma unroll
  for (int k = 0; k < kMaxK; ++k)
#pragma unroll
    for (int c = 0; c < C; ++c) dw[k][c] = 0.f;
  const IO* __restrict__ xb = x + (size_t)b * p.T * p.D + ch;
  const IO* __restrict__ gb = dy + (size_t)b * p.T * p.D + ch;
  IO* __restrict__ ob = dx + (size_t)b * p.T * p.D + ch;
  float x1[C], x2[C], x3[C], g1[C], g2[C], g3[C];  // previous inputs; previous three dy
#pragma unroll
  for (int c = 0; c < C; ++c) x1[c] = x2[c] = x3[c] = g1[c] = g2[c] = g3[c] = 0.f;
  if (first - 1 >= 0) load_n<IO, C>(xb + (size_t)(first - 1) * p.D, x1);
  if (first - 2 >= 0) load_n<IO, C>(xb + (size_t)(first - 2) * p.D, x2);
  if (first - 3 >= 0) load_n<IO, C>(xb + (size_t)(first - 3) * p.D, x3);
  auto emit = [&](int t, const float (&g0)[C]) {  // dx[t-3] = w0 dy[t-3] + w1 dy[t-2] + w2 dy[t-1] + w3 dy[t]
    if (t - 3 >= first && t - 3 < p.T) {
      float o[C];
#pragma unroll
      for (int c = 0; c < C; ++c) o[c] = wk[0][c] * g3[c] + wk[1][c] * g2[c] + wk[2][c] * g1[c] + wk[3][c] * g0[c];
      store_n<IO, C>(ob + (size_t)(t - 3) * p.D, o);
    }
#pragma unroll
    for (int c = 0; c < C; ++c) { g3[c] = g2[c]; g2[c] = g1[c]; g1[c] = g0[c]; }
  };
  auto loaded = [&](const IO* src, int t, float (&v)[C]) {  // clamped address, masked
    load_n<IO, C>(src + (size_t)min(t, p.T - 1) * p.D, v);
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = t < p.T ? v[c] : 0.f;
  };
  int t0 = first;
  for (; t0 < min(p.T, first + p.runs * kRun); t0 += kRun) {
#pragma unroll
    for (int r = 0; r < kRun; ++r) {
      float x0[C], g0[C];
      loaded(gb, t0 + r, g0);
      loaded(xb, t0 + r, x0);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        dw[0][c] = fmaf(x0[c], g0[c], dw[0][c]);
        dw[1][c] = fmaf(x1[c], g0[c], dw[1][c]);
        dw[2][c] = fmaf(x2[c], g0[c], dw[2][c]);
        dw[3][c] = fmaf(x3[c], g0[c], dw[3][c]);
        x3[c] = x2[c]; x2[c] = x1[c]; x1[c] = x0[c];
      }
      emit(t0 + r, g0);
    }
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {  // the three steps behind, for dx alone
    float g0[C];
    loaded(gb, t0 + r, g0);
    emit(t0 + r, g0);
  }
  float* dst = dwp + ((size_t)(b * gridDim.y + blockIdx.y) * kMaxK) * p.D + ch;
#pragma unroll
  for (int k = 0; k < kMaxK; ++k) store_n<float, C>(dst + (size_t)k * p.D, dw[k]);
}
// Column sums of partial rows.  K > 0: columns are [k][d] and the result is stored as [d][K] (k < K only).
template <bool TALL>
__global__ void __launch_bounds__(kSumThreads<TALL>) m3b_colsum_kernel(const float* __restrict__ part, int rows, int n,
                                                                       float* __restrict__ out, int D, int K) {
  begin_dependent();
  const int j0 = blockIdx.x * kSumCols<TALL>, mine = j0 + threadIdx.x % kSumCols<TALL>;
  col_sum<TALL>(part + mine, rows, n, mine < n, [&](int c, float t) {
    const int j = j0 + c, k = j / D, d = j % D;
    if (j >= n) return;
    if (K == 0) out[j] = t;
    else if (k < K) out[(size_t)d * K + k] = t;
  });
}

// sum over the LN lanes of a group; the mask names only the caller's group (the lane groups of a warp may run different numbers
// of loop iterations)
template <int LN>
__device__ __forceinline__ float group_sum(float v) {
  const unsigned mask = ((1u << LN) - 1u) << (threadIdx.x & 31 & ~(LN - 1));
#pragma unroll
  for (int o = LN / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

// ------------------------------------------------------------------ B / C: RMSNorm over N + bias
// grid (ctas, G, 2) x 128: blockIdx.z selects b or c, blockIdx.y the group; a group of LN lanes per row (b, t), the smallest
// power of two with 8 LN >= N.  N <= 128, N % 8 == 0.  (16 lanes for every N: rows of 16 states left 14 of 16 lanes idle, 4096 x
// 4 groups forward / backward 11.2 / 18.8 us, 3.9 / 6.8 now.)
template <typename IO>
struct BcArgs {
  const IO* x[2];
  const float* scale[2];
  const float* bias[2];
  IO* y[2];
  const IO* dy[2];
  IO* dx[2];
  float* part[2];  // [ctas][G][2][N]: dscale, dbias partial rows
  float *dscale[2], *dbias[2];
};
template <typename IO, int LN>
__global__ void __launch_bounds__(128) m3b_bc_fwd_kernel(BlkP p, BcArgs<IO> a) {
  begin_dependent();
  constexpr int ROWS = 128 / LN;
  const int which = blockIdx.z, g = blockIdx.y, ln = threadIdx.x % LN, grp = threadIdx.x / LN;
  const bool act = ln * 8 < p.N;
  float sc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, bi[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (act) { load8<float>(a.scale[which] + ln * 8, sc); load8<float>(a.bias[which] + g * p.N + ln * 8, bi); }
  const size_t nbt = (size_t)p.B * p.T;
  for (size_t bt = (size_t)blockIdx.x * ROWS + grp; bt < nbt; bt += (size_t)gridDim.x * ROWS) {
    const size_t off = (bt * p.G + g) * p.N + ln * 8;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (act) load8<IO>(a.x[which] + off, v);
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) ss = fmaf(v[c], v[c], ss);
    ss = group_sum<LN>(ss);
    const float rn = rsqrtf(ss / (float)p.N + p.eps);
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = fmaf(v[c] * rn, sc[c], bi[c]);
    if (act) store8<IO>(a.y[which] + off, v);
  }
}
template <typename IO, int LN>
__global__ void __launch_bounds__(128) m3b_bc_bwd_kernel(BlkP p, BcArgs<IO> a) {
  begin_dependent();
  constexpr int ROWS = 128 / LN;
  __shared__ float red[ROWS][2][8 * LN];
  const int which = blockIdx.z, g = blockIdx.y, ln = threadIdx.x % LN, grp = threadIdx.x / LN;
  const bool act = ln * 8 < p.N;
  float sc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float ds[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, db[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (act) load8<float>(a.scale[which] + ln * 8, sc);
  const size_t nbt = (size_t)p.B * p.T;
  for (size_t bt = (size_t)blockIdx.x * ROWS + grp; bt < nbt; bt += (size_t)gridDim.x * ROWS) {
    const size_t off = (bt * p.G + g) * p.N + ln * 8;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, gy[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (act) { load8<IO>(a.x[which] + off, v); load8<IO>(a.dy[which] + off, gy); }
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      ss = fmaf(v[c], v[c], ss);
      dot = fmaf(v[c], gy[c] * sc[c], dot);
    }
    ss = group_sum<LN>(ss);
    dot = group_sum<LN>(dot);
    const float rn = rsqrtf(ss / (float)p.N + p.eps);
    const float k2 = rn * rn * dot / (float)p.N;
    float o[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      ds[c] = fmaf(gy[c], v[c] * rn, ds[c]);
      db[c] += gy[c];
      o[c] = rn * (gy[c] * sc[c] - v[c] * k2);
    }
    if (act) store8<IO>(a.dx[which] + off, o);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) { red[grp][0][ln * 8 + c] = ds[c]; red[grp][1][ln * 8 + c] = db[c]; }
  __syncthreads();
  float* dst = a.part[which] + ((size_t)(blockIdx.x * p.G + g) * 2) * p.N;
  for (int i = threadIdx.x; i < 2 * p.N; i += 128) {
    const int kind = i / p.N, c = i % p.N;
    float s = 0.f;
#pragma unroll 8
    for (int k = 0; k < ROWS; ++k) s += red[k][kind][c];
    dst[(size_t)kind * p.N + c] = s;
  }
}
// The sums of the partial rows of b and c in one launch.  grid (ceil(N/16), G + 1, 2): dbias of group y, or (y == G) dscale,
// which is the sum over the groups too.
template <typename IO>
__global__ void __launch_bounds__(kSumThreads<true>) m3b_bc_sum_kernel(BlkP p, BcArgs<IO> a, int ctas) {
  begin_dependent();
  const int which = blockIdx.z, g = blockIdx.y, c0 = blockIdx.x * kSumCols<true>, mine = c0 + threadIdx.x % kSumCols<true>;
  const bool scale = g == p.G;
  const size_t row = 2 * (size_t)p.N;
  const float* part = a.part[which] + (scale ? 0 : g * row + p.N) + mine;
  float* out = scale ? a.dscale[which] : a.dbias[which] + g * p.N;
  col_sum<true>(part, scale ? (size_t)ctas * p.G : ctas, scale ? row : p.G * row, mine < p.N, [&](int c, float t) {
    if (c0 + c < p.N) out[c0 + c] = t;
  });
}

// ------------------------------------------------------------------ post: RMSNorm over D x SiLU gate
// Rows of up to 512 channels: a warp per token row, 16 bytes of a row per lane and piece, no barrier.  (A CTA per row of 448 float32
// channels had 56 of 256 threads at work and three barriers a row: 4096 rows forward / backward 11.2 / 17.4 us, 6.5 / 11.9
// now.  The backward spills 56 bytes at two CTAs an SM; with one, 8 x 4096 rows of 512 bf16 channels take 46 us for 35.)
constexpr int kWarpRow = 512;
template <typename IO>
struct WarpRow {
  static constexpr int C = 16 / sizeof(IO), NV = kWarpRow / (32 * C);  // channels of a piece, pieces of a lane
  int ch[NV];
  bool act[NV];
  __device__ explicit WarpRow(int D) {
#pragma unroll
    for (int x = 0; x < NV; ++x) {
      ch[x] = C * ((threadIdx.x & 31) + 32 * x);
      act[x] = ch[x] < D;
    }
  }
  template <typename T>
  __device__ void load(const T* row, float (&v)[NV][C]) const {
#pragma unroll
    for (int x = 0; x < NV; ++x) {
      if (act[x]) {
        load_n<T, C>(row + ch[x], v[x]);
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) v[x][c] = 0.f;
      }
    }
  }
  __device__ void store(IO* row, const float (&v)[NV][C]) const {
#pragma unroll
    for (int x = 0; x < NV; ++x)
      if (act[x]) store_n<IO, C>(row + ch[x], v[x]);
  }
};
template <typename IO>
__global__ void __launch_bounds__(256) m3b_post_fwd_warp_kernel(BlkP p, const IO* __restrict__ y, const IO* __restrict__ z,
                                                                const float* __restrict__ wn, IO* __restrict__ out) {
  begin_dependent();
  using R = WarpRow<IO>;
  const R r(p.D);
  float w[R::NV][R::C];
  r.load(wn, w);
  const size_t rows = (size_t)p.B * p.T;
  for (size_t row = blockIdx.x * 8 + (threadIdx.x >> 5); row < rows; row += (size_t)gridDim.x * 8) {
    float yv[R::NV][R::C], zv[R::NV][R::C];
    r.load(y + row * p.D, yv);
    r.load(z + row * p.D, zv);
    float ss = 0.f;
#pragma unroll
    for (int x = 0; x < R::NV; ++x)
#pragma unroll
      for (int c = 0; c < R::C; ++c) ss = fmaf(yv[x][c], yv[x][c], ss);
    const float rn = rsqrtf(warp_sum(ss) / (float)p.D + p.eps);
#pragma unroll
    for (int x = 0; x < R::NV; ++x)
#pragma unroll
      for (int c = 0; c < R::C; ++c) yv[x][c] = yv[x][c] * rn * w[x][c] * zv[x][c] * sigmoid_f(zv[x][c]);
    r.store(out + row * p.D, yv);
  }
}
template <typename IO>
__global__ void __launch_bounds__(256, 2) m3b_post_bwd_warp_kernel(BlkP p, const IO* __restrict__ y, const IO* __restrict__ z,
                                                                const float* __restrict__ wn, const IO* __restrict__ dout,
                                                                IO* __restrict__ dy, IO* __restrict__ dz,
                                                                float* __restrict__ dwp) {
  begin_dependent();
  using R = WarpRow<IO>;
  __shared__ float red[8][kWarpRow];
  const R r(p.D);
  float w[R::NV][R::C], dw[R::NV][R::C];
  r.load(wn, w);
#pragma unroll
  for (int x = 0; x < R::NV; ++x)
#pragma unroll
    for (int c = 0; c < R::C; ++c) dw[x][c] = 0.f;
  const size_t rows = (size_t)p.B * p.T;
  const int warp = threadIdx.x >> 5;
  for (size_t row = blockIdx.x * 8 + warp; row < rows; row += (size_t)gridDim.x * 8) {
    float yv[R::NV][R::C], zv[R::NV][R::C], gv[R::NV][R::C], g[R::NV][R::C];
    r.load(y + row * p.D, yv);
    r.load(z + row * p.D, zv);
    r.load(dout + row * p.D, gv);
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int x = 0; x < R::NV; ++x)
#pragma unroll
      for (int c = 0; c < R::C; ++c) {
        g[x][c] = gv[x][c] * (zv[x][c] * sigmoid_f(zv[x][c])) * w[x][c];
        ss = fmaf(yv[x][c], yv[x][c], ss);
        dot = fmaf(yv[x][c], g[x][c], dot);
      }
    ss = warp_sum(ss);
    dot = warp_sum(dot);
    const float rn = rsqrtf(ss / (float)p.D + p.eps), k2 = rn * rn * dot / (float)p.D;
#pragma unroll
    for (int x = 0; x < R::NV; ++x)
#pragma unroll
      for (int c = 0; c < R::C; ++c) {
        const float sg = sigmoid_f(zv[x][c]), sz = zv[x][c] * sg, yn = yv[x][c] * rn;
        dw[x][c] = fmaf(gv[x][c] * sz, yn, dw[x][c]);
        zv[x][c] = gv[x][c] * w[x][c] * yn * fmaf(sz, 1.f - sg, sg);
        g[x][c] = rn * (g[x][c] - yv[x][c] * k2);
      }
    r.store(dy + row * p.D, g);
    r.store(dz + row * p.D, zv);
  }
#pragma unroll
  for (int x = 0; x < R::NV; ++x)
#pragma unroll
    for (int c = 0; c < R::C; ++c) red[warp][r.ch[x] + c] = dw[x][c];
  __syncthreads();
  for (int d = threadIdx.x; d < p.D; d += 256) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += red[k][d];
    dwp[(size_t)blockIdx.x * p.D + d] = s;
  }
}
// Wider rows: a CTA of 256 threads per token row (D <= 2048, D % 8 == 0), grid-stride over the B*T rows
__device__ __forceinline__ float cta_sum(float v, float* red) {
  v = warp_sum(v);
  __syncthreads();  // red may still be read from the previous use
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += red[k];
  return s;
}
template <typename IO>
__global__ void __launch_bounds__(256) m3b_post_fwd_kernel(BlkP p, const IO* __restrict__ y, const IO* __restrict__ z,
                                                           const float* __restrict__ wn, IO* __restrict__ out) {
  begin_dependent();
  __shared__ float red[8];
  const int ch = threadIdx.x * 8;
  const bool act = ch < p.D;
  float w[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (act) load8<float>(wn + ch, w);
  const size_t rows = (size_t)p.B * p.T;
  for (size_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t off = row * p.D + ch;
    float yv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, zv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (act) { load8<IO>(y + off, yv); load8<IO>(z + off, zv); }
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) ss = fmaf(yv[c], yv[c], ss);
    ss = cta_sum(ss, red);
    const float rn = rsqrtf(ss / (float)p.D + p.eps);
#pragma unroll
    for (int c = 0; c < 8; ++c) yv[c] = yv[c] * rn * w[c] * zv[c] * sigmoid_f(zv[c]);
    if (act) store8<IO>(out + off, yv);
  }
}
template <typename IO>
__global__ void __launch_bounds__(256) m3b_post_bwd_kernel(BlkP p, const IO* __restrict__ y, const IO* __restrict__ z,
                                                           const float* __restrict__ wn, const IO* __restrict__ dout,
                                                           IO* __restrict__ dy, IO* __restrict__ dz,
                                                           float* __restrict__ dwp) {
  begin_dependent();
  __shared__ float red[8];
  const int ch = threadIdx.x * 8;
  const bool act = ch < p.D;
  float w[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, dw[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (act) load8<float>(wn + ch, w);
  const size_t rows = (size_t)p.B * p.T;
  for (size_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t off = row * p.D + ch;
    float yv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, zv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float gv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (act) { load8<IO>(y + off, yv); load8<IO>(z + off, zv); load8<IO>(dout + off, gv); }
    float ss = 0.f, dot = 0.f, g[8], sz[8], dsz[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float sg = sigmoid_f(zv[c]);
      sz[c] = zv[c] * sg;
      dsz[c] = fmaf(sz[c], 1.f - sg, sg);
      g[c] = gv[c] * sz[c] * w[c];
      ss = fmaf(yv[c], yv[c], ss);
      dot = fmaf(yv[c], g[c], dot);
    }
    ss = cta_sum(ss, red);
    dot = cta_sum(dot, red);
    const float rn = rsqrtf(ss / (float)p.D + p.eps);
    const float k2 = rn * rn * dot / (float)p.D;
    float dzv[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float yn = yv[c] * rn;
      dw[c] = fmaf(gv[c] * sz[c], yn, dw[c]);
      dzv[c] = gv[c] * w[c] * yn * dsz[c];
      g[c] = rn * (g[c] - yv[c] * k2);
    }
    if (act) { store8<IO>(dy + off, g); store8<IO>(dz + off, dzv); }
  }
  if (act) store8<float>(dwp + (size_t)blockIdx.x * p.D + ch, dw);
}

}  // namespace m3b

// ------------------------------------------------------------------ host
using m3b::BlkP;

static BlkP make_m3b(const mxb_mamba3_desc* d, int K, float eps) {
  BlkP p{};
  p.B = d->B; p.T = d->T; p.D = d->D; p.N = d->N; p.G = d->G; p.K = K; p.eps = eps;
  return p;
}
bool mamba3_block_supported(const mxb_mamba3_desc* d) {
  return d->D % 8 == 0 && d->D <= 2048 && d->N % 8 == 0 && d->N <= 128 && d->G > 0;
}
// Steps of a lane of the convolution, in units of kRun: up to four while that gives three CTAs an SM.  A CTA of bf16 rows with up to
// sixteen lanes has little under way, and what takes the time is the chain of steps: rounds of the CTAs that the GPU holds at once
// (five an SM by the forward's registers) times the steps of a lane, the fewest.  Forward, us, 444 x 67 x 64 channels 11.6 by the
// first rule, 7.7 by the second; 16 x 4096 x 32 17.3 and 11.3.  (float32 rows have twice the lanes and gain nothing over both passes.)
static int m3b_run_units(const mxb_mamba3_desc* d) {
  const bool f32 = d->io_dtype == MXB_F32;
  const int lanes = d->D / (f32 ? m3b::kConvC<float> : m3b::kConvC<m3b::bf16>);
  auto ctas = [&](int u) { return (size_t)d->B * ((lanes + 127) / 128) * ((d->T + u * m3b::kRun - 1) / (u * m3b::kRun)); };
  int u = 4;
  if (f32 || lanes > 16) {
    while (u > 1 && ctas(u) < 3 * 148) u /= 2;
    return u;
  }
  auto chain = [&](int units) {
    const size_t at_once = 148 * 5;
    return (ctas(units) + at_once - 1) / at_once * std::min(units * m3b::kRun, (int)d->T);
  };
  for (int v : {2, 1})
    if (chain(v) < chain(u)) u = v;
  return u;
}
static int m3b_runs(const mxb_mamba3_desc* d) {
  const int steps = m3b::kRun * m3b_run_units(d);
  return (d->T + steps - 1) / steps;
}
static int m3b_bc_lanes(const mxb_mamba3_desc* d) {
  int n = 2;
  while (8 * n < d->N) n *= 2;
  return n;
}
static int m3b_bc_ctas(const mxb_mamba3_desc* d) {
  const size_t per = 128 / m3b_bc_lanes(d), want = ((size_t)d->B * d->T + per - 1) / per;
  return (int)std::min<size_t>(want, 148 * 4);
}
// CTAs of the output stage: what is on the GPU at once by the registers of the kernels (bf16 and float32: rows of a warp 70 and 73
// forward, 128 backward; wider ones 48 and 47, 80 backward; 256 threads).
static int m3b_post_ctas(const mxb_mamba3_desc* d, bool bwd) {
  const size_t rows = (size_t)d->B * d->T;
  if (d->D <= m3b::kWarpRow) return (int)std::min<size_t>((rows + 7) / 8, 148 * (bwd ? 2 : 3));
  return (int)std::min<size_t>(rows, 148 * (bwd ? 3 : 5));
}
size_t mamba3_block_workspace_bytes(const mxb_mamba3_desc* d) {
  const size_t conv = (size_t)d->B * m3b_runs(d) * m3b::kMaxK * d->D * sizeof(float);
  const size_t bc = 2 * (size_t)m3b_bc_ctas(d) * d->G * 2 * d->N * sizeof(float);
  const size_t post = (size_t)m3b_post_ctas(d, true) * d->D * sizeof(float);
  size_t m = conv > bc ? conv : bc;
  m = m > post ? m : post;
  return m + 256;
}

static void m3b_colsum(const float* part, int rows, int n, float* out, int D, int K, cudaStream_t st) {
  auto launch = [&](auto tall) {
    constexpr bool TALL = decltype(tall)::value;
    MXB_LAUNCH("m3b_colsum_kernel", st,
               (launch_kernel(m3b::m3b_colsum_kernel<TALL>, (n + kSumCols<TALL> - 1) / kSumCols<TALL>, kSumThreads<TALL>, 0, st, part, rows, n, out, D, K)));
  };
  if (col_sum_tall(n)) launch(std::true_type{});
  else launch(std::false_type{});
}

template <typename IO>
static mxb_status m3b_conv(const mxb_mamba3_desc* d, int K, const void* x, const float* w, void* y, const void* dy,
                           void* dx, float* dw, void* ws, cudaStream_t st) {
  BlkP p = make_m3b(d, K, 0.f);
  p.runs = m3b_run_units(d);
  p.wvec = K == 4 && reinterpret_cast<uintptr_t>(w) % 16 == 0;
  const int c = dy ? m3b::kConvBwdC : m3b::kConvC<IO>;
  const dim3 grid((d->D / c + 127) / 128, m3b_runs(d), d->B);
  if (!dy) {
    MXB_LAUNCH("m3b_conv_fwd_kernel", st,
               (launch_kernel(m3b::m3b_conv_fwd_kernel<IO>, grid, 128, 0, st, p, static_cast<const IO*>(x), w, static_cast<IO*>(y))));
    return check_launch("m3b_conv_fwd");
  }
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + 256);
  MXB_LAUNCH("m3b_conv_bwd_kernel", st,
             (launch_kernel(m3b::m3b_conv_bwd_kernel<IO>, grid, 128, 0, st, p, static_cast<const IO*>(x), w, static_cast<const IO*>(dy),
                                                                 static_cast<IO*>(dx), part)));
  const int rows = d->B * m3b_runs(d), n = m3b::kMaxK * d->D;
  m3b_colsum(part, rows, n, dw, d->D, K, st);
  return check_launch("m3b_conv_bwd");
}
mxb_status mamba3_block_conv(const mxb_mamba3_desc* d, int K, const void* x, const float* w, void* y, const void* dy,
                             void* dx, float* dw, void* ws, cudaStream_t st) {
  return d->io_dtype == MXB_F32 ? m3b_conv<float>(d, K, x, w, y, dy, dx, dw, ws, st)
                                : m3b_conv<m3b::bf16>(d, K, x, w, y, dy, dx, dw, ws, st);
}

template <typename F>
static void by_lanes(const mxb_mamba3_desc* d, F&& f) {
  switch (m3b_bc_lanes(d)) {
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    case 8: f(std::integral_constant<int, 8>{}); break;
    default: f(std::integral_constant<int, 16>{}); break;
  }
}
template <typename IO>
static mxb_status m3b_bc(const mxb_mamba3_desc* d, float eps, const void* bp, const void* cp, const float* bs,
                         const float* cs, const float* bb, const float* cb, void* b, void* c, const void* db,
                         const void* dc, void* dbp, void* dcp, float* dbs, float* dcs, float* dbb, float* dcb, void* ws,
                         cudaStream_t st) {
  BlkP p = make_m3b(d, 0, eps);
  m3b::BcArgs<IO> a{};
  a.x[0] = static_cast<const IO*>(bp); a.x[1] = static_cast<const IO*>(cp);
  a.scale[0] = bs; a.scale[1] = cs; a.bias[0] = bb; a.bias[1] = cb;
  const int ctas = m3b_bc_ctas(d);
  const dim3 grid(ctas, d->G, 2);
  if (!db) {
    a.y[0] = static_cast<IO*>(b); a.y[1] = static_cast<IO*>(c);
    by_lanes(d, [&](auto ln) {
      MXB_LAUNCH("m3b_bc_fwd_kernel", st, (launch_kernel(m3b::m3b_bc_fwd_kernel<IO, decltype(ln)::value>, grid, 128, 0, st, p, a)));
    });
    return check_launch("m3b_bc_fwd");
  }
  a.dy[0] = static_cast<const IO*>(db); a.dy[1] = static_cast<const IO*>(dc);
  a.dx[0] = static_cast<IO*>(dbp); a.dx[1] = static_cast<IO*>(dcp);
  a.dscale[0] = dbs; a.dscale[1] = dcs; a.dbias[0] = dbb; a.dbias[1] = dcb;
  a.part[0] = reinterpret_cast<float*>(static_cast<char*>(ws) + 256);
  a.part[1] = a.part[0] + (size_t)ctas * d->G * 2 * d->N;
  by_lanes(d, [&](auto ln) {
    MXB_LAUNCH("m3b_bc_bwd_kernel", st, (launch_kernel(m3b::m3b_bc_bwd_kernel<IO, decltype(ln)::value>, grid, 128, 0, st, p, a)));
  });
  MXB_LAUNCH("m3b_bc_sum_kernel", st,
             (launch_kernel(m3b::m3b_bc_sum_kernel<IO>, dim3((d->N + kSumCols<true> - 1) / kSumCols<true>, d->G + 1, 2),
                            kSumThreads<true>, 0, st, p, a, ctas)));
  return check_launch("m3b_bc_bwd");
}
mxb_status mamba3_block_bc(const mxb_mamba3_desc* d, float eps, const void* bp, const void* cp, const float* bs,
                           const float* cs, const float* bb, const float* cb, void* b, void* c, const void* db,
                           const void* dc, void* dbp, void* dcp, float* dbs, float* dcs, float* dbb, float* dcb, void* ws,
                           cudaStream_t st) {
  return d->io_dtype == MXB_F32
             ? m3b_bc<float>(d, eps, bp, cp, bs, cs, bb, cb, b, c, db, dc, dbp, dcp, dbs, dcs, dbb, dcb, ws, st)
             : m3b_bc<m3b::bf16>(d, eps, bp, cp, bs, cs, bb, cb, b, c, db, dc, dbp, dcp, dbs, dcs, dbb, dcb, ws, st);
}

template <typename IO>
static mxb_status m3b_post(const mxb_mamba3_desc* d, float eps, const void* y, const void* z, const float* wn, void* out,
                           const void* dout, void* dy, void* dz, float* dwn, void* ws, cudaStream_t st) {
  BlkP p = make_m3b(d, 0, eps);
  const int ctas = m3b_post_ctas(d, dout != nullptr);
  const bool narrow = d->D <= m3b::kWarpRow;
  const IO *yv = static_cast<const IO*>(y), *zv = static_cast<const IO*>(z);
  if (!dout) {
    MXB_LAUNCH("m3b_post_fwd_kernel", st,
               (launch_kernel(narrow ? m3b::m3b_post_fwd_warp_kernel<IO> : m3b::m3b_post_fwd_kernel<IO>, ctas, 256, 0, st, p, yv, zv, wn,
                              static_cast<IO*>(out))));
    return check_launch("m3b_post_fwd");
  }
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + 256);
  MXB_LAUNCH("m3b_post_bwd_kernel", st,
             (launch_kernel(narrow ? m3b::m3b_post_bwd_warp_kernel<IO> : m3b::m3b_post_bwd_kernel<IO>, ctas, 256, 0, st, p, yv, zv, wn,
                            static_cast<const IO*>(dout), static_cast<IO*>(dy), static_cast<IO*>(dz), part)));
  m3b_colsum(part, ctas, d->D, dwn, d->D, 0, st);
  return check_launch("m3b_post_bwd");
}
mxb_status mamba3_block_post(const mxb_mamba3_desc* d, float eps, const void* y, const void* z, const float* wn, void* out,
                             const void* dout, void* dy, void* dz, float* dwn, void* ws, cudaStream_t st) {
  return d->io_dtype == MXB_F32 ? m3b_post<float>(d, eps, y, z, wn, out, dout, dy, dz, dwn, ws, st)
                                : m3b_post<m3b::bf16>(d, eps, y, z, wn, out, dout, dy, dz, dwn, ws, st);
}

}  // namespace mxb
