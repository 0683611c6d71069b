// Shared declarations of the Mamba-3 channel kernels (serial walk: mamba3.cu, window-parallel: mamba3_windows.cu).
#pragma once

#include "common.cuh"

namespace mxb {

constexpr int kM3Window = 16;  // checkpoint spacing of the serial walk

struct M3P {
  int B, T, D, N, G, NH, Kp, nW;
  int LPC;  // lanes per channel: 32, or 16 / 8 where d_state <= 32 / 16 would leave most lanes of a warp without a state pair
  const void *x, *b, *c;
  const float *dt, *lam, *theta, *a_log;
  void* y;
  float *ck_h, *ck_phi;  // checkpoints [B,nW,D,N], [B,nW,D,Kp]
  const void* dy;
  void* dx;
  float *ddt, *dlam, *dtheta, *da_log;
  void *db, *dc;
  // channel kernels: CW channels (warps) per CTA, S = channels per group / CW slices per group
  int CW, S;
  float *pb32, *pc32;  // [B,T,G,S,N] rows summed over the CW channels of a CTA
  float* hd;           // head-broadcast layout only: per-channel ddt, dlam, dtheta, 3 x [B,T,D]
  float* dal_part;     // per-batch (window-parallel: per batch and window) da_log: [.,D,N], or [.,D] head-broadcast
  // window-parallel kernels (mamba3_windows.cu)
  int w0;              // first window of a launch
  int vec;             // rows of b, c, theta can be read two state pairs at a time
  float *dtv, *lamv;   // softplus(dt), sigmoid(lambda) in the layout of dt, lambda
  float* dtsum;        // [B,nW,D] sum of dt over the window
  float* dhk;          // [B,nW,D,N]: dh entering the window from later steps
  float* ang;          // [B,nW,D,Kp]: angle-gradient sum of the window, then of all later windows
};

__device__ __forceinline__ float m3_softplus(float x) {
  if (x > 20.f) return x;
  if (x < -20.f) return expf(x);
  return log1pf(expf(x));
}
__device__ __forceinline__ float m3_sigmoid(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float m3_wrap(float phi) {
  // Cody-Waite reduction by 2 pi = 6.28125 + 1.9353071795864769e-3
  const float k = rintf(phi * 0.15915494309189535f);
  phi = fmaf(-k, 6.28125f, phi);
  return fmaf(-k, 1.9353071795864769e-3f, phi);
}

// Sum over the LPC lanes that share a channel (LPC = 32: the whole warp); every lane of the group gets the sum.
template <int LPC>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = LPC / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct M3Idx {
  int D, N, G, NH, Kp, cpg, cph;
  __device__ explicit M3Idx(const M3P& p) : M3Idx(p, p.NH) {}
  __device__ M3Idx(const M3P& p, int nh) : D(p.D), N(p.N), G(p.G), NH(nh), Kp(p.Kp), cpg(p.D / p.G), cph(nh > 0 ? p.D / nh : 1) {}
  __device__ size_t chan(size_t row, int d) const { return NH > 0 ? row * NH + d / cph : row * D + d; }
  __device__ size_t theta(size_t row, int d, int kp) const {
    return NH > 0 ? row * NH + d / cph : (row * D + d) * Kp + kp;
  }
  __device__ size_t alog(int d, int n) const { return NH > 0 ? (size_t)(d / cph) : (size_t)d * N + n; }
  __device__ size_t grp(size_t row, int d, int n) const { return (row * G + d / cpg) * N + n; }
};

// Sums of the partials the reverse walks leave, in a fixed order, by the block-th of `blocks` blocks.
// dB, dC: rows over the slices of a group.
template <typename IO>
__device__ __forceinline__ void m3_bc_sum(const M3P& p, int block, int blocks) {
  const size_t total = (size_t)p.B * p.T * p.G * p.N;
  for (size_t i = block * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)blocks * blockDim.x) {
    const size_t r = i / p.N;
    const int n = (int)(i - r * p.N);
    float sb = 0.f, sc = 0.f;
    for (int s = 0; s < p.S; ++s) {
      sb += p.pb32[(r * p.S + s) * p.N + n];
      sc += p.pc32[(r * p.S + s) * p.N + n];
    }
    static_cast<IO*>(p.db)[i] = from_f32<IO>(sb);
    static_cast<IO*>(p.dc)[i] = from_f32<IO>(sc);
  }
}
inline int m3_bc_sum_blocks(const M3P& p, int threads) {
  const size_t want = ((size_t)p.B * p.T * p.G * p.N + threads - 1) / threads, most = 148 * 2048 / threads;
  return (int)(want < most ? want : most);
}
// da_log over the batch (and windows: `rows`), and the channels of a head; 32 outputs a block of 16 warps, each with a slice.
constexpr int kDalogSlices = 16;
__device__ __forceinline__ void m3_dalog_sum(const M3P& p, int rows, int block) {
  __shared__ float red[kDalogSlices][32];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, i = block * 32 + lane;
  const int cph = p.NH > 0 ? p.D / p.NH : 1, outs = p.NH > 0 ? p.NH : p.D * p.N, total = rows * cph;
  float s = 0.f;
  if (i < outs) {
#pragma unroll 8
    for (int r = slice; r < total; r += kDalogSlices)
      s += p.NH > 0 ? p.dal_part[(size_t)(r / cph) * p.D + i * cph + r % cph] : p.dal_part[(size_t)r * outs + i];
  }
  red[slice][lane] = s;
  __syncthreads();
  if (slice == 0 && i < outs) {
    s = 0.f;
#pragma unroll
    for (int k = 0; k < kDalogSlices; ++k) s += red[k][lane];
    p.da_log[i] = s;
  }
}
inline int m3_dalog_blocks(const M3P& p) { return ((p.NH > 0 ? p.NH : p.D * p.N) + 31) / 32; }

constexpr int kM3WinSteps = 8;  // steps per window of the window-parallel kernels
struct M3WinShape { int lanes, warps; };  // lanes per channel; warps per CTA, all of one group
M3WinShape m3w_shape(const M3P& p);
mxb_status m3w_forward(const M3P& p, bool f32, cudaStream_t st);
mxb_status m3w_backward(const M3P& p, bool f32, bool have_states, cudaStream_t st);

}  // namespace mxb
