// Mamba-3 selective scan in chunked dual ("SSD") form on tensor cores - head-broadcast
// layout (dt, lambda, theta per (b,t,head), A per head), head dim 64, d_state 128, bf16 I/O.
//
// With scalar decay per (step, head) the exponential-trapezoidal recurrence
//     h_t = alpha_t h_{t-1} + gamma_t Brot_t x_t^T + beta_t Brot_{t-1} x_{t-1}^T ,  y_t = Crot_t^T h_t
// (reference: gpu/cuda_kernels/mamba3_selective_scan_fwd_v2_emit.cu:65-115) has the closed form
//     y_t = sum_{s<=t} (Crot_t . Brot_s) exp(Lam_t - Lam_s) w_ts x_s ,   Lam = cumsum(dt A),
//     w_ts = e_s = gamma_s + (1-lambda_{s+1}) dt_{s+1}  for s < t,   w_tt = gamma_t,
// because beta_{s+1} exp(Lam_t - Lam_{s+1}) = (1-lambda_{s+1}) dt_{s+1} exp(Lam_t - Lam_s).  Per chunk of
// 64 steps (M_ts = exp(Lam_t-Lam_s) w_ts [s<=t], r_s = exp(Lam_end - Lam_s), L = exp(Lam_end)):
//     Y  = (Crot Brot^T * M) X + diag(exp(Lam)) Crot H0          H1 = L H0 + Brot^T diag(r e) X
// so the only sequential part is the elementwise chunk scan H1 = L H0 + Hc.  The backward is the
// hand-derived adjoint of these two lines (checked against float64 autograd of the recurrence
// before it was written); its sequential part is the mirrored scan dH0 = L dH1 + Dc.
//
//   m3s_scalars_kernel      per chunk: dt, lambda, the chunk's share of the angle (fp64)
//   m3s_angle_prefix_kernel (long sequences) the shares to the sums over the chunks in front
//   m3s_chunk_scalars_kernel per chunk: decay sums, trapezoid weights, sines/cosines of the cumulative angle (one record)
//   m3s_state_pass_kernel   per (b, head), sequential over the chunks, forward or reverse: the chunk contribution
//                           Brot^T diag(r e) X (or Crot^T diag(exp(Lam)) dY) folded into the running state
//   m3s_chunk_out_kernel    per chunk: Y
//   m3s_scan_out_kernel     the forward state pass and Y in one kernel, where the (batch, head) pairs fill the GPU
//   m3s_chunk_grad_kernel   per chunk and up to 16 heads of a group: dx, dB, dC summed over these heads, per-token scalars
//   m3s_tail_kernel         per chunk: ddt, dlambda, dtheta, da_log shares; dB, dC summed over the CTAs of a group
#include <cuda.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "mma_sync.cuh"
#include "packed.cuh"
#include "umma_tiles.cuh"

namespace mxb {
namespace m3s {

constexpr int Q = 64;    // chunk
constexpr int P = 64;    // head dim
constexpr int N = 128;   // d_state
using bf16 = __nv_bfloat16;
using tc::mbar_arrive;
using tc::pack8;
using tc::unpack8;

struct SsdP {
  int B, T, D, G, NH, n;   // n = chunks
  int splits, hp;          // CTAs of the chunk-gradient kernel per group of heads, heads of each (the last one may have fewer)
  int no_tma;              // stage operands with cp.async even where tensor maps can be made
  const bf16 *x, *b, *c, *dy;
  const float *dt_raw, *lam_raw, *theta, *a_log;
  bf16 *y, *dx;
  float *ddt, *dlam, *dtheta, *da_log;
  int* status;
  // workspace
  float *dt, *lam, *theta_t;    // [B,NH,T]
  bf16 *H0, *dH1;               // [B,NH,n,N,P] state at chunk start / state gradient at chunk end
  float *dphi, *da, *de, *dgam; // [B,NH,T] per-token scalar gradients (dphi: of the angle increment of a step)
  float* dal_part;              // [B,n,NH] shares of da_log
  float* cs;                    // [B,NH,n] ChunkScal records
  bf16 *pb, *pc;                // [B,G*splits,n] column-blocked [64][128] images: partial dB, dC (summed in fp32 by the tail kernel)
};

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : (x < -20.f ? expf(x) : log1pf(expf(x))); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ void sts16(uint8_t* base, uint32_t off, uint4 v) { *reinterpret_cast<uint4*>(base + off) = v; }
__device__ __forceinline__ void ld_acc32(uint32_t taddr, int warp, int c0, float (&f)[32]) {
  uint32_t r[32];
  tc::tmem_ld_32x32b_x32(taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, r);
  tc::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void ld_acc16(uint32_t taddr, int warp, int c0, float (&f)[16]) {
  uint32_t r[16];
  tc::tmem_ld_32x32b_x16(taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, r);
  tc::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(r[i]);
}

// 8 columns of a result as four pairs.
__device__ __forceinline__ void ld_pairs(uint32_t taddr, int warp, f2 (&f)[4]) {
  uint32_t r[8];
  tc::tmem_ld_32x32b_x8(taddr + ((uint32_t)(32 * (warp & 3)) << 16), r);
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}
__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Two packed bf16 as two floats and back.
__device__ __forceinline__ f2 widen2(uint32_t w) { return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ uint32_t narrow2(f2 v) {
  const float2 t = unpack2(v);
  return tc::pack_bf16(t.x, t.y);
}
__device__ __forceinline__ f2 neg2(f2 v) { return v ^ 0x8000000080000000ull; }

// Per-chunk scalars: computed once per (batch, head, chunk) by m3s_chunk_scalars_kernel into a workspace record
// and fetched by every chunk kernel with its operand tiles (the record is a whole number of 16-byte units).
struct ChunkScal {
  float Lam[Q];   // in-chunk inclusive cumulative sum of dt A
  float gam[Q];   // lambda dt
  float e[Q];     // gam_s + (1 - lambda_{s+1}) dt_{s+1}
  float sn[Q], cs[Q];  // sine / cosine of the cumulative rotation angle
  float dexp[Q];  // exp(Lam)
  float r[Q];     // exp(Lam_last - Lam)
  float re[Q];    // r e
  float L, A, pad[2];
};
static_assert(sizeof(ChunkScal) % 16 == 0, "record moves in 16-byte units");
constexpr int kScalUnits = sizeof(ChunkScal) / 16;

// PREFIX: share has the sum over the chunks in front (m3s_angle_prefix_kernel) instead of the chunk's own.
template <bool PREFIX>
__global__ void __launch_bounds__(64) m3s_chunk_scalars_kernel(SsdP p, const double* share) {
  begin_dependent();
  __shared__ __align__(16) ChunkScal s;
  __shared__ float sdt[Q];
  __shared__ double wsum[4];
  const int tid = threadIdx.x, c = blockIdx.x, head = blockIdx.y, b = blockIdx.z, t0 = c * Q;
  const size_t base = ((size_t)b * p.NH + head) * p.T;
  const size_t ci = ((size_t)b * p.NH + head) * p.n + c;
  const float A = -expf(p.a_log[head]);
  {
    const int t = t0 + tid;
    const bool ok = t < p.T;
    const float dt = ok ? p.dt[base + t] : 0.f, lam = ok ? p.lam[base + t] : 0.f;
    const float nxt = (t + 1 < p.T) ? (1.f - p.lam[base + t + 1]) * p.dt[base + t + 1] : 0.f;
    sdt[tid] = dt;
    s.gam[tid] = lam * dt;
    s.e[tid] = lam * dt + nxt;
    // cumulative rotation angle in fp64: the shares of the chunks in front, then the steps of this one
    double before = 0.0, phi = ok ? (double)dt * (double)p.theta_t[base + t] : 0.0;
    if (PREFIX) {
      if (tid == 0) before = share[((size_t)b * p.n + c) * p.NH + head];
    } else {
      for (int x = tid; x < c; x += Q) before += share[((size_t)b * p.n + x) * p.NH + head];
    }
    const int lane = tid & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, phi, o);
      if (lane >= o) phi += up;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 31) {
      wsum[tid >> 5] = before;
      wsum[2 + (tid >> 5)] = phi;
    }
    __syncthreads();
    phi += wsum[0] + wsum[1] + (tid >= 32 ? wsum[2] : 0.0);
    const double two_pi = 6.283185307179586476925, inv_two_pi = 1.0 / two_pi;
    float sn = 0.f, cs = 1.f;
    if (ok) sincosf((float)(phi - two_pi * rint(phi * inv_two_pi)), &sn, &cs);  // wrapped to [-pi, pi]
    s.sn[tid] = sn; s.cs[tid] = cs;
  }
  __syncthreads();
  if (tid < 32) {  // inclusive in-chunk cumulative sum of a = dt A, two per lane
    const float a0 = sdt[2 * tid] * A, a1 = sdt[2 * tid + 1] * A;
    float v = a0 + a1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, v, o);
      if (tid >= o) v += t;
    }
    s.Lam[2 * tid] = v - a1;
    s.Lam[2 * tid + 1] = v;
  }
  __syncthreads();
  {
    const float last = s.Lam[Q - 1];
    const float r = __expf(last - s.Lam[tid]);
    s.dexp[tid] = __expf(s.Lam[tid]);
    s.r[tid] = r;
    s.re[tid] = r * s.e[tid];
    if (tid == 0) { s.L = __expf(last); s.A = A; s.pad[0] = s.pad[1] = 0.f; }
  }
  __syncthreads();
  uint4* dst = reinterpret_cast<uint4*>(p.cs + ci * (sizeof(ChunkScal) / 4));
  for (int u = tid; u < kScalUnits; u += 64) dst[u] = reinterpret_cast<const uint4*>(&s)[u];
}
// cp.async of the record of chunk ci into shared memory (part of the caller's current cp.async group)
__device__ __forceinline__ void issue_chunk_scalars(const SsdP& p, size_t ci, ChunkScal& s) {
  const uint32_t sd = tc::smem_u32(&s);
  const float* src = p.cs + ci * (sizeof(ChunkScal) / 4);
  for (int u = threadIdx.x; u < kScalUnits; u += blockDim.x) tc::cp_async16(sd + 16 * u, src + 4 * u);
}

// ---- asynchronous staging: raw cp.async copies into the blocked layout, then in-place fix-ups ----
// With t = 8 (u / 128) + u % 8 and c8 = (u / 8) % 16 the unit of a [64][128] tile sits at byte 16 u, and
// likewise for [.][64] tiles with t = 8 (u / 64) + u % 8, c8 = (u / 8) % 8: eight consecutive lanes fill one
// 128-byte row group (no bank conflicts) and read 64-byte pieces of a row.
__device__ __forceinline__ void issue_rows_tile(uint8_t* dst, const bf16* src, const SsdP& p, int b, int g, int t0) {
  const uint32_t sd = tc::smem_u32(dst);
  for (int u = threadIdx.x; u < Q * 16; u += blockDim.x) {
    const int t = ((u >> 7) << 3) | (u & 7), c8 = (u >> 3) & 15;
    const bool ok = t0 + t < p.T;
    tc::cp_async16(sd + 16 * u, ok ? src + (((size_t)b * p.T + t0 + t) * p.G + g) * N + c8 * 8 : src, ok);
  }
}
__device__ __forceinline__ void issue_x_tile(uint8_t* dst, const bf16* src, const SsdP& p, int b, int d0, int t0) {
  const uint32_t sd = tc::smem_u32(dst);
  for (int u = threadIdx.x; u < Q * 8; u += blockDim.x) {
    const int t = ((u >> 6) << 3) | (u & 7), c8 = (u >> 3) & 7;
    const bool ok = t0 + t < p.T;
    tc::cp_async16(sd + 16 * u, ok ? src + ((size_t)b * p.T + t0 + t) * p.D + d0 + c8 * 8 : src, ok);
  }
}
// Rows of a token tensor ([B,T,heads,64] or a 64-column slab of [B,T,G,128]) into a swizzled slab, by threads tid of nt;
// src: the row of step t0.
__device__ __forceinline__ void stage_slab(uint32_t dst, const bf16* src, int T, size_t stride, int t0, int tid, int nt) {
  for (int u = tid; u < Q * 8; u += nt) {
    const int t = u >> 3, c8 = u & 7;
    const bool ok = t0 + t < T;
    tc::cp_async16(dst + (uint32_t)t * 128u + (uint32_t)((c8 ^ (t & 7)) << 4), ok ? src + (size_t)t * stride + c8 * 8 : src, ok);
  }
}
// [128 n][64 p] bf16 state saved by the state pass as the byte image of the blocked tile
__device__ __forceinline__ void issue_state_tile(uint8_t* dst, const bf16* src) {
  const uint32_t sd = tc::smem_u32(dst);
  for (int u = threadIdx.x; u < N * 8; u += blockDim.x) tc::cp_async16(sd + 16 * u, src + 8 * u);
}
// Rotates the (even, odd) pairs of every row of a landed [64][128] tile in place.
__device__ __forceinline__ void rotate_tile(uint8_t* tile, const float* sn, const float* cs) {
  for (int u = threadIdx.x; u < Q * 16; u += blockDim.x) {
    const int t = ((u >> 7) << 3) | (u & 7);
    float e[8];
    unpack8(*reinterpret_cast<const uint4*>(tile + 16 * u), e);
    const float s_ = sn[t], c_ = cs[t];
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const float ev = e[k], od = e[k + 1];
      e[k] = fmaf(c_, ev, s_ * od);
      e[k + 1] = fmaf(c_, od, -(s_ * ev));
    }
    *reinterpret_cast<uint4*>(tile + 16 * u) = pack8(e);
  }
}
// ---- the same fix-ups and views for tiles that the copy engine wrote with 128-byte swizzle (SW = true) ----
template <bool SW>
__device__ __forceinline__ uint32_t in_unit(int t, int c8, int W) {
  return SW ? tc::sw128_unit(t, c8) : tc::kmajor_unit(t, c8, W);
}
template <bool SW>
__device__ __forceinline__ tc::Tile in_kmajor(const void* ptr, int W) {
  return SW ? tc::kmajor_sw128_tile(ptr, 8192) : tc::kmajor_tile(ptr, W);
}
template <bool SW>
__device__ __forceinline__ tc::Tile in_mnmajor(const void* ptr, int W) {
  return SW ? tc::mnmajor_sw128_tile(ptr, 8192) : tc::mnmajor_tile(ptr, W);
}
// A thread keeps to one row (rows of eight lanes start in eight different banks through the swizzle), so a row's sine and cosine
// are read once; two pairs of states share a packed register, even and odd states apart.  nt threads, a multiple of 64.
template <bool SW>
__device__ __forceinline__ void rotate_in_tile(uint8_t* tile, const float* sn, const float* cs, int tid, int nt) {
  if constexpr (!SW) {
    rotate_tile(tile, sn, cs);
  } else {
    const int t = tid & 63, per = 1024 / nt, c0 = (tid >> 6) * per;
    const f2 c2 = dup2(cs[t]), s2 = dup2(sn[t]), n2 = dup2(-sn[t]);
    auto rot = [&](uint32_t& a, uint32_t& b) {
      const f2 e = pack2(__uint_as_float(a << 16), __uint_as_float(b << 16));
      const f2 o = pack2(__uint_as_float(a & 0xffff0000u), __uint_as_float(b & 0xffff0000u));
      const float2 x = unpack2(mad2(c2, e, mul2(s2, o))), y = unpack2(mad2(c2, o, mul2(n2, e)));
      a = tc::pack_bf16(x.x, y.x);
      b = tc::pack_bf16(x.y, y.y);
    };
#pragma unroll
    for (int q0 = 0; q0 < per; q0 += 4) {  // four units, all loads before the first store
      uint4 raw[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) raw[q] = *reinterpret_cast<const uint4*>(tile + tc::sw128_unit(t, c0 + q0 + q));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        rot(raw[q].x, raw[q].y);
        rot(raw[q].z, raw[q].w);
        *reinterpret_cast<uint4*>(tile + tc::sw128_unit(t, c0 + q0 + q)) = raw[q];
      }
    }
  }
}
// Rows of a [64][64] tile (swizzled) times a factor each, bf16 again; src and dst may be the same.
__device__ __forceinline__ void scale_rows(uint8_t* dst, const uint8_t* src, const float* factor, int tid, int nt) {
  const int t = tid & 63, per = 512 / nt, c0 = (tid >> 6) * per;
  const f2 f = dup2(factor[t]);
#pragma unroll
  for (int q = 0; q < per; ++q) {
    const uint32_t at = tc::sw128_unit(t, c0 + q);
    const uint4 x = *reinterpret_cast<const uint4*>(src + at);
    *reinterpret_cast<uint4*>(dst + at) = make_uint4(narrow2(mul2(widen2(x.x), f)), narrow2(mul2(widen2(x.y), f)),
                                                     narrow2(mul2(widen2(x.z), f)), narrow2(mul2(widen2(x.w), f)));
  }
}
// G*M of row t and the 32 columns from n0 on: M_ts = exp(Lam_t - Lam_s) e_s below the diagonal, gam_t on it.
__device__ __forceinline__ void mask_row(float (&g)[32], const ChunkScal& s, int t, int n0) {
  const float gt = s.gam[t];
  const f2 lt = dup2(s.Lam[t]), minus = dup2(-1.f), log2e = dup2(1.4426950408889634f);
  const int k = t - n0;
#pragma unroll
  for (int x = 0; x < 8; ++x) {  // branch-free, so the exponentials of different columns overlap
    const ulonglong2 l4 = *reinterpret_cast<const ulonglong2*>(s.Lam + n0 + 4 * x);
    const float4 e4 = *reinterpret_cast<const float4*>(s.e + n0 + 4 * x);
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const int q = 4 * x + 2 * y;
      const float2 d = unpack2(mad2(y ? l4.y : l4.x, minus, lt));
      const float2 a = unpack2(mul2(pack2(fminf(d.x, 0.f), fminf(d.y, 0.f)), log2e));
      const f2 w = pack2(q < k ? (y ? e4.z : e4.x) : gt, q + 1 < k ? (y ? e4.w : e4.y) : gt);
      const float2 r = unpack2(mul2(pack2(g[q], g[q + 1]), mul2(pack2(ex2(a.x), ex2(a.y)), w)));
      g[q] = q <= k ? r.x : 0.f;
      g[q + 1] = q + 1 <= k ? r.y : 0.f;
    }
  }
}

struct ChunkMaps {
  CUtensorMap b, c;   // [B,T,G,128] viewed as (N, G, T, B), boxes of 64 columns x 64 steps, 128-byte swizzle
  CUtensorMap x, dy, dx;  // [B,T,heads,64] viewed as (P, heads, T, B)
};

// ------------------------------------------------------------ per-token scalars
constexpr int kScalThreads = 256;
constexpr int kScalHeads = 8;    // heads of a block: 32 bytes of a step, so that a small call still spreads over SMs

// dt, lambda and theta of a chunk's steps and up to 8 heads, from the caller's [B,T,heads] to rows of [B,heads,T] through shared
// memory (whole sectors on both sides), and the chunk's share of the rotation angle, in fp64, into `share` [B,n,heads].
__global__ void __launch_bounds__(kScalThreads) m3s_scalars_kernel(SsdP p, double* share) {
  begin_dependent();
  __shared__ float dr[Q][kScalHeads + 1], lr[Q][kScalHeads + 1], th[Q][kScalHeads + 1];
  __shared__ double wsum[2 * kScalHeads];
  // (chunks and groups of heads share the x axis: the others end at 65,535)
  const int groups = (p.NH + kScalHeads - 1) / kScalHeads, c = blockIdx.x / groups, b = blockIdx.y;
  const int h0 = blockIdx.x % groups * kScalHeads, nh = min(kScalHeads, p.NH - h0), t0 = c * Q, nt = min(Q, p.T - t0);
  const int tid = threadIdx.x;
  if (blockIdx.x == 0 && b == 0 && tid < 64) p.status[tid] = 0;  // (the kernels behind this one raise it)
  const size_t row0 = ((size_t)b * p.T + t0) * p.NH + h0;
#pragma unroll
  for (int x = 0; x < Q * kScalHeads / kScalThreads; ++x) {
    const int u = tid + x * kScalThreads, t = u / kScalHeads, h = u % kScalHeads;
    const bool in = t < nt && h < nh;
    const size_t r = in ? row0 + (size_t)t * p.NH + h : row0;
    dr[t][h] = __ldg(p.dt_raw + r);
    lr[t][h] = __ldg(p.lam_raw + r);
    th[t][h] = __ldg(p.theta + r);
  }
  __syncthreads();
#pragma unroll
  for (int x = 0; x < Q * kScalHeads / kScalThreads; ++x) {
    const int u = tid + x * kScalThreads, h = u / Q, t = u % Q;
    double inc = 0.0;
    if (t < nt && h < nh) {
      const size_t o = ((size_t)b * p.NH + h0 + h) * p.T + t0 + t;
      const float dt = softplus_f(dr[t][h]), theta = th[t][h];
      p.dt[o] = dt;
      p.lam[o] = sigmoid_f(lr[t][h]);
      p.theta_t[o] = theta;
      inc = (double)dt * (double)theta;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) inc += __shfl_xor_sync(0xffffffffu, inc, o);  // (a warp has 32 steps of one head)
    if ((tid & 31) == 0) wsum[u >> 5] = inc;
  }
  __syncthreads();
  if (tid < nh) share[((size_t)b * p.n + c) * p.NH + h0 + tid] = wsum[2 * tid] + wsum[2 * tid + 1];
}

// The chunks' shares of the angle to the sums of the shares in front of them, in place: a thread adds a segment of the chunks of
// one head, the segments are scanned in shared memory, and the thread goes through its segment again.  Eight heads a block, so
// that a row of shares is read by whole sectors.
constexpr int kPrefixSegs = 128;
__global__ void __launch_bounds__(kScalHeads * kPrefixSegs) m3s_angle_prefix_kernel(SsdP p, double* share) {
  begin_dependent();
  __shared__ double sums[kPrefixSegs][kScalHeads];
  const int seg = threadIdx.x / kScalHeads, hl = threadIdx.x % kScalHeads, head = blockIdx.x * kScalHeads + hl;
  const int len = (p.n + kPrefixSegs - 1) / kPrefixSegs, c0 = min(seg * len, p.n), c1 = head < p.NH ? min(c0 + len, p.n) : c0;
  double* col = share + (size_t)blockIdx.y * p.n * p.NH + head;
  double sum = 0.0;
#pragma unroll 8
  for (int c = c0; c < c1; ++c) sum += col[(size_t)c * p.NH];
  sums[seg][hl] = sum;
  __syncthreads();
#pragma unroll
  for (int o = 1; o < kPrefixSegs; o <<= 1) {
    const double up = seg >= o ? sums[seg - o][hl] : 0.0;
    __syncthreads();
    sums[seg][hl] += up;
    __syncthreads();
  }
  double before = seg > 0 ? sums[seg - 1][hl] : 0.0;
#pragma unroll 8
  for (int c = c0; c < c1; ++c) {
    const double own = col[(size_t)c * p.NH];
    col[(size_t)c * p.NH] = before;
    before += own;
  }
}

// ------------------------------------------------------------ state pass
// One CTA per (batch, head) walks the chunks in order (mode 0) or in reverse (mode 1) and keeps the running
// state in registers (thread = state row n and 32 of its 64 fp32 columns):
//   mode 0: H0_c = H;  H = L_c H + Brot_c^T diag(r e) X_c          (states at chunk start, for y and the backward)
//   mode 1: dH1_c = dH; dH = L_c dH + Crot_c^T diag(exp(Lam)) dY_c  (state gradients at chunk end)
// The chunk contribution is one M=128 tcgen05 tile that never leaves the SM.  The saved state goes from registers to the byte
// image of the [128][64] operand tile (eight rows of a unit column are one 128-byte line).
//
// Only the update of the state is sequential, so everything before it runs ahead: a warp issues the copies, four warps rotate
// and scale landed tiles in place, a warp issues the products into two accumulators by turns, eight warps hold the state,
// fold in an accumulator and store the state (one sequence of 32 heads x 64 chunks: 57 us a pass, chunk by chunk in one group
// of warps 84; 8 sequences 101, where it is the arithmetic of the rotation that counts, 107 before a thread kept to a row).  Every hand-over is an mbarrier with a bounded wait; a warp whose wait has run out stops waiting and working but goes through its loop.
// NS stages in flight: three and four warps that prepare tiles where two CTAs share an SM, six and eight where one has it.
template <int NS>
constexpr int kPassPrep = NS == 3 ? 4 : 8;
template <int NS>
constexpr int kPassThreads = 32 * (10 + kPassPrep<NS>);
template <int NS>
constexpr int kPassSmem = NS * (16384 + 8192) + (NS + 2) * (int)sizeof(ChunkScal) + (4 * NS + 12) * 8 + 16 + 1024;

struct PassMaps {
  CUtensorMap r;  // b or c: [B,T,G,128] viewed as (N, G, T, B), boxes of 64 columns x 64 steps, 128-byte swizzle
  CUtensorMap x;  // x or dy: [B,T,heads,64] viewed as (P, heads, T, B)
};

// TMA = true: the three operand boxes of a chunk arrive by the copy engine; TMA = false: cp.async staging into the same
// swizzled positions.
template <bool TMA, int NS>
__global__ void __launch_bounds__(kPassThreads<NS>, NS == 3 ? 2 : 1) m3s_state_pass_kernel(SsdP p, int mode, const __grid_constant__ PassMaps maps) {
  begin_dependent();
  constexpr int NC = NS + 2;         // scalar records: the decay is read behind the product
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Rt = sm;                  // xNS [64 s][128 n] B or C rows, rotated in place
  uint8_t* Xt = Rt + NS * 16384;     // xNS [64 s][64 p] x or dy, scaled in place
  ChunkScal* scal = reinterpret_cast<ChunkScal*>(Xt + NS * 8192);
  uint64_t* full = reinterpret_cast<uint64_t*>(scal + NC);  // xNS: tiles landed
  uint64_t* ready = full + NS;       // xNS: tiles rotated and scaled
  uint64_t* freed = ready + NS;      // xNS: product done
  uint64_t* accfull = freed + NS;    // x2: product done
  uint64_t* accfree = accfull + 2;   // x2: accumulator read
  uint64_t* cfree = accfree + 2;       // xNC: scalar record read
  uint32_t* tslot = reinterpret_cast<uint32_t*>(cfree + NC);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.x, b = blockIdx.y, n = p.n;
  const int d0 = head * P, g = d0 / (p.D / p.G);
  const size_t cbase = ((size_t)b * p.NH + head) * n;
  auto chunk_at = [&](int it) { return mode == 0 ? it : n - 1 - it; };
  if (warp == 0) { tc::tmem_alloc(tslot, 128); tc::tmem_relinquish(); }
  if (tid == 32) {
    for (int s = 0; s < NS; ++s) { tc::mbar_init(full + s, TMA ? 1 : 33); tc::mbar_init(ready + s, kPassPrep<NS>); tc::mbar_init(freed + s, 1); }
    for (int s = 0; s < 2; ++s) { tc::mbar_init(accfull + s, 1); tc::mbar_init(accfree + s, 8); }
    for (int s = 0; s < NC; ++s) tc::mbar_init(cfree + s, 8);
    tc::mbar_fence_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  bool ok = true;
  auto wait = [&](uint64_t* m, int parity) { if (ok) ok = tc::mbar_wait(m, (uint32_t)parity & 1u); };
  auto arrive = [&](uint64_t* m) {
    __syncwarp();
    if (lane == 0) mbar_arrive(m);
  };
  if (warp == 8) {          // ---- copies
    int issued = 0;
    for (int it = 0; it < n; ++it) {
      const int s = it % NS, c = chunk_at(it);
      if (it >= NS) wait(freed + s, it / NS - 1);
      if (it >= NC) wait(cfree + it % NC, it / NC - 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ++issued;
      if (lane == 0) {
        tc::mbar_expect_tx(full + s, (TMA ? 16384 + 8192 : 0) + (uint32_t)sizeof(ChunkScal));
        if (TMA) {
          tc::tma_load_4d(tc::smem_u32(Rt + s * 16384), &maps.r, 0, g, c * Q, b, full + s);
          tc::tma_load_4d(tc::smem_u32(Rt + s * 16384) + 8192, &maps.r, 64, g, c * Q, b, full + s);
          tc::tma_load_4d(tc::smem_u32(Xt + s * 8192), &maps.x, 0, head, c * Q, b, full + s);
        }
        tc::bulk_load(tc::smem_u32(scal + it % NC), p.cs + (cbase + c) * (sizeof(ChunkScal) / 4), (uint32_t)sizeof(ChunkScal), full + s);
      }
      if (!TMA) {
        const size_t row = (size_t)b * p.T + c * Q;
        const bf16* rsrc = (mode == 0 ? p.b : p.c) + (row * p.G + g) * N;
        for (int sl = 0; sl < 2; ++sl)
          stage_slab(tc::smem_u32(Rt + s * 16384) + 8192 * sl, rsrc + 64 * sl, p.T, (size_t)p.G * N, c * Q, lane, 32);
        stage_slab(tc::smem_u32(Xt + s * 8192), (mode == 0 ? p.x : p.dy) + row * p.D + d0, p.T, p.D, c * Q, lane, 32);
        tc::cp_async_wait_all();
        tc::fence_async_smem();
        mbar_arrive(full + s);
      }
    }
    for (int q = max(0, issued - NS); q < issued; ++q) tc::mbar_wait(full + q % NS, (q / NS) & 1);  // (outlive the copies)
  } else if (warp == 9) {   // ---- products
    if (tc::elect_one()) {
      for (int it = 0; it < n; ++it) {
        const int s = it % NS, a = it & 1;
        wait(ready + s, it / NS);
        if (it > 1) wait(accfree + a, (it >> 1) - 1);
        if (!ok) break;
        tc::fence_after_sync();
        // [128 n x 64 p] = R^T X, both contracted over their rows
        tc::issue_gemm(taddr + 64 * a, tc::mnmajor_sw128_tile(Rt + s * 16384, 8192), tc::mnmajor_sw128_tile(Xt + s * 8192, 8192), 128, P, Q, false);
        tc::mma_commit(accfull + a);
        tc::mma_commit(freed + s);
      }
    }
    __syncwarp();
  } else if (warp >= 10) {  // ---- rows rotated, x or dy scaled
    const int u0 = tid - 320;
    for (int it = 0; it < n; ++it) {
      const int st = it % NS;
      wait(full + st, it / NS);
      const ChunkScal& s = scal[it % NC];
      rotate_in_tile<true>(Rt + st * 16384, s.sn, s.cs, u0, 32 * kPassPrep<NS>);
      scale_rows(Xt + st * 8192, Xt + st * 8192, mode == 0 ? s.re : s.dexp, u0, 32 * kPassPrep<NS>);
      tc::fence_async_smem();
      arrive(ready + st);
    }
  } else if (warp < 8) {    // ---- the state: thread = state row and 32 of its 64 columns
    const int nrow = tid & 127, half = tid >> 7;
    f2 H[16];
#pragma unroll
    for (int x = 0; x < 16; ++x) H[x] = 0ull;
    uint4* out = reinterpret_cast<uint4*>((mode == 0 ? p.H0 : p.dH1) + cbase * (N * P)) + (tc::kmajor_unit(nrow, 4 * half, P) >> 4);
    for (int it = 0; it < n; ++it) {
      const int a = it & 1;
#pragma unroll
      for (int x = 0; x < 4; ++x) out[(size_t)chunk_at(it) * (N * P / 8) + 8 * x] =
          make_uint4(narrow2(H[4 * x]), narrow2(H[4 * x + 1]), narrow2(H[4 * x + 2]), narrow2(H[4 * x + 3]));
      wait(accfull + a, it >> 1);
      tc::fence_after_sync();
      ok = __all_sync(0xffffffffu, ok);
      const f2 L = dup2(scal[it % NC].L);
      if (ok) {
        f2 f[16];
#pragma unroll
        for (int q = 0; q < 4; ++q) ld_pairs(taddr + 64 * a + 32 * half + 8 * q, warp, *reinterpret_cast<f2(*)[4]>(f + 4 * q));
        tc::tmem_ld_wait();
#pragma unroll
        for (int x = 0; x < 16; ++x) H[x] = mad2(L, H[x], f[x]);
      }
      tc::fence_before_sync();
      arrive(accfree + a);
      arrive(cfree + it % NC);
    }
  }
  if (!ok && lane == 0) atomicExch(p.status, 11);
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 128);
}

// ------------------------------------------------------------ chunk output
// A CTA is a chain of dependent steps, so the kernel is sized for FOUR CTAs per SM: 64 TMEM columns (weight-stationary
// products: every thread has a row and half of the columns of a result) and 51 KB of shared memory.  The chunk state H0
// lands in the Brot tile once G = Crot Brot^T has been formed (its copy hides behind the mask epilogue), and Crot H0
// joins the second MMA batch.  Bound by shared memory (the copies, the rotation in place and the operand reads move
// about 200 KB per chunk): 8 x 4096 x 32 heads 194 us with half of the lanes idle in the epilogues, 185 now; 256 threads
// per CTA 188.
constexpr int kOutSmem = 16384 * 2 + 8192 * 2 + sizeof(ChunkScal) + 64 + 1024;

template <bool TMA>
__global__ void __launch_bounds__(128, 4) m3s_chunk_out_kernel(SsdP p, const __grid_constant__ ChunkMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Bt = sm;               // [64][128] Brot, then [128][64] H0
  uint8_t* Ct = Bt + 16384;       // [64][128] Crot
  uint8_t* Ht = Bt;
  uint8_t* Xt = Ct + 16384;       // [64][64]  x
  uint8_t* Gm = Xt + 8192;        // [64][64]  (Crot Brot^T) * M
  ChunkScal& s = *reinterpret_cast<ChunkScal*>(Gm + 8192);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(&s + 1);  // [0] MMA completion, [1] token tiles landed, [2] H0 landed
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 3);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x, head = blockIdx.y, b = blockIdx.z, t0 = c * Q;
  const int d0 = head * P, g = d0 / (p.D / p.G);
  const size_t ci = ((size_t)b * p.NH + head) * p.n + c;

  if (warp == 0) { tc::tmem_alloc(tslot, 64); tc::tmem_relinquish(); }
  // the thread that initialises the barriers also issues the copies, on another warp than the TMEM allocation
  if (tid == 32) {
    for (int m = 0; m < 3; ++m) tc::mbar_init(mbar + m, 1);
    tc::mbar_fence_init();
  }
  bool ok = true;
  if (TMA) {  // every operand by the copy engine
    if (tid == 32) {
      tc::mbar_expect_tx(mbar + 1, 2 * 16384 + 8192 + (uint32_t)sizeof(ChunkScal));
      for (int sl = 0; sl < 2; ++sl) {
        tc::tma_load_4d(tc::smem_u32(Bt) + 8192 * sl, &maps.b, 64 * sl, g, t0, b, mbar + 1);
        tc::tma_load_4d(tc::smem_u32(Ct) + 8192 * sl, &maps.c, 64 * sl, g, t0, b, mbar + 1);
      }
      tc::tma_load_4d(tc::smem_u32(Xt), &maps.x, 0, head, t0, b, mbar + 1);
      tc::bulk_load(tc::smem_u32(&s), p.cs + ci * (sizeof(ChunkScal) / 4), (uint32_t)sizeof(ChunkScal), mbar + 1);
    }
    __syncthreads();  // barriers initialised before anyone waits on them
    ok = tc::mbar_wait(mbar + 1, 0);
  } else {
    issue_rows_tile(Bt, p.b, p, b, g, t0);
    issue_rows_tile(Ct, p.c, p, b, g, t0);
    issue_x_tile(Xt, p.x, p, b, d0, t0);
    issue_chunk_scalars(p, ci, s);
    tc::cp_async_commit();
    tc::cp_async_wait<0>();
  }
  __syncthreads();
  rotate_in_tile<TMA>(Bt, s.sn, s.cs, tid, 128);
  rotate_in_tile<TMA>(Ct, s.sn, s.cs, tid, 128);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  if (tid == 0) {
    tc::issue_gemm<true>(taddr, in_kmajor<TMA>(Ct, N), in_kmajor<TMA>(Bt, N), 64, Q, N, false);           // G = Crot Brot^T
    tc::mma_commit(mbar);
  }
  if (ok) ok = tc::mbar_wait(mbar, 0);
  tc::fence_after_sync();
  // Brot is dead: the chunk state takes its place while the mask is applied
  if (TMA) {
    if (tid == 32) {
      tc::mbar_expect_tx(mbar + 2, 16384);
      tc::bulk_load(tc::smem_u32(Ht), p.H0 + ci * (N * P), 16384, mbar + 2);
    }
  } else {
    issue_state_tile(Ht, p.H0 + ci * (N * P));
    tc::cp_async_commit();
  }
  // weight-stationary products: this thread's row, and the half of the columns it holds of every result
  const int t = 32 * (warp & 1) + lane, n0 = 32 * (warp >> 1);
  if (ok) {
    float f[32];
    ld_acc32(taddr, warp, 0, f);
    mask_row(f, s, t, n0);
#pragma unroll
    for (int x = 0; x < 4; ++x) sts16(Gm, tc::kmajor_unit(t, (n0 >> 3) + x, Q), pack8(&f[8 * x]));
  }
  if (TMA) { if (ok) ok = tc::mbar_wait(mbar + 2, 0); }  // H0
  else tc::cp_async_wait<0>();
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (ok && tid == 0) {
    tc::issue_gemm<true>(taddr, tc::kmajor_tile(Gm, Q), in_mnmajor<TMA>(Xt, P), 64, P, Q, false);  // (G*M) X, over the consumed G
    tc::issue_gemm<true>(taddr + 32, in_kmajor<TMA>(Ct, N), tc::mnmajor_tile(Ht, P), 64, P, N, false);    // Crot H0
    tc::mma_commit(mbar);
  }
  if (ok) ok = tc::mbar_wait(mbar, 1);
  tc::fence_after_sync();
  if (ok) {  // y = (G*M) X + exp(Lam) Crot H0, assembled over the x tile (dead) and written out in full rows
    const float de = s.dexp[t];
    float f[32], f2[32];
    ld_acc32(taddr, warp, 0, f);
    ld_acc32(taddr + 32, warp, 0, f2);
#pragma unroll
    for (int jj = 0; jj < 32; ++jj) f[jj] = fmaf(de, f2[jj], f[jj]);
#pragma unroll
    for (int x = 0; x < 4; ++x) sts16(Xt, tc::kmajor_unit(t, (n0 >> 3) + x, P), pack8(&f[8 * x]));
  } else if (tid == 0) {
    atomicExch(p.status, 12);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (ok) {
    for (int u = tid; u < Q * 8; u += 128) {  // 64-byte row pieces, conflict-free shared-memory reads
      const int r = ((u >> 6) << 3) | (u & 7), c8 = (u >> 3) & 7;
      if (t0 + r < p.T)
        *reinterpret_cast<uint4*>(p.y + ((size_t)b * p.T + t0 + r) * p.D + d0 + c8 * 8) =
            *reinterpret_cast<const uint4*>(Xt + 16 * u);
    }
  }
  if (warp == 0) tc::tmem_dealloc(taddr, 64);
}

// ------------------------------------------------------------ states and output in one pass
// The forward state pass with the chunk output behind it: one CTA per (batch, head) walks the chunks, and what the output of a
// chunk needs (the rotated rows of B, x and the state in front of the chunk) is on the SM already, so B and x are read and B is
// rotated once and the state is not read back.  The same products, roundings and order of sums as m3s_state_pass_kernel and
// m3s_chunk_out_kernel: the same bits.
//
// 512 threads and 110 KB, two CTAs per SM.  Warps 0-3 hold the state (thread = row, 64 columns) and write its image, which the
// product with Crot reads and, for a backward, a bulk store keeps; warps 4-7 mask G and put y together; warps 8-11 rotate B and
// C and scale x; the last four issue copies, state products, output products and stores.  Hand-overs are mbarriers with bounded
// waits.  A wait cannot miss its phase: a stage is loaded again only when y and the scalars of its chunk are through, so what
// is counted per stage stays within two chunks, and of every other barrier the next phase needs its waiters to have passed.
// G*M takes the place of Brot, y that of x.
// TMEM: the state's contribution [0, 64) and [64, 128) by turns, G [128, 160), Crot H0 [160, 192), (G*M) X [192, 224).
// No unit is at its limit (5 x 2048 x 32 heads: 25 % of the issue slots, shared memory 29 %, tensor pipe 8 %, DRAM 14 %): what takes
// the time is the chain of hand-overs of a chunk (rotation, product, state; G, mask, product, y) with two CTAs an SM to fill it.
// 8 x 4096 x 32 heads 222 us where the two kernels take 102 + 184 (without keeping the states 200).
constexpr int kScanThreads = 512;
constexpr int kScanStage = 2 * 16384 + 8192;
constexpr int kScanSmem = 2 * kScanStage + 8192 + 16384 + 2 * (int)sizeof(ChunkScal) + 21 * 8 + 16 + 1024;
static_assert(2 * (kScanSmem + 1024) <= 228 * 1024, "two CTAs per SM");

struct ScanMaps {
  CUtensorMap b, c;  // as in ChunkMaps
  CUtensorMap x, y;
};

__global__ void __launch_bounds__(kScanThreads, 2) m3s_scan_out_kernel(SsdP p, int save, const __grid_constant__ ScanMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Xs = sm + 2 * kScanStage;   // [64][64] r e x (swizzled like x); a stage: B, C, x
  uint8_t* Ht = Xs + 8192;             // [128][64] state in front of the chunk, operand image
  ChunkScal* scal = reinterpret_cast<ChunkScal*>(Ht + 16384);  // x2
  uint64_t* full = reinterpret_cast<uint64_t*>(scal + 2);      // x2: a chunk's operands landed
  uint64_t* sfree = full + 2;          // x2: y has left, the scalars are read
  uint64_t* accfull = sfree + 2;       // x2: product of the state (Brot and r e x are no longer needed)
  uint64_t* accfree = accfull + 2;     // x2: accumulator read
  uint64_t* readyb = accfree + 2;      // x2: Brot and r e x written
  uint64_t* readyc = readyb + 2;       // x2: Crot written
  uint64_t* yready = readyc + 2;       // x2: y written
  uint64_t* xsfree = yready + 2;       // r e x read
  uint64_t* hready = xsfree + 1;       // image of the state written
  uint64_t* hfree = hready + 1;        // ... and read, by the product and the store
  uint64_t* gfull = hfree + 1;         // G
  uint64_t* gmready = gfull + 1;       // G*M written
  uint64_t* yfull = gmready + 1;       // both products of y
  uint64_t* yfree = yfull + 1;         // ... and read
  uint32_t* tslot = reinterpret_cast<uint32_t*>(yfree + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.x, b = blockIdx.y, n = p.n;
  const int g = head * P / (p.D / p.G);
  const size_t cbase = ((size_t)b * p.NH + head) * n;
  constexpr uint32_t tG = 128, tH = 160, tY = 192;
  if (warp == 0) { tc::tmem_alloc(tslot, 256); tc::tmem_relinquish(); }
  if (tid == 32) {
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(full + s, 1); tc::mbar_init(sfree + s, 5);
      tc::mbar_init(accfull + s, 1); tc::mbar_init(accfree + s, 4);
      tc::mbar_init(readyb + s, 4); tc::mbar_init(readyc + s, 4); tc::mbar_init(yready + s, 4);
    }
    tc::mbar_init(xsfree, 1); tc::mbar_init(hready, 4); tc::mbar_init(hfree, 2);
    tc::mbar_init(gfull, 1); tc::mbar_init(gmready, 4); tc::mbar_init(yfull, 1); tc::mbar_init(yfree, 4);
    tc::mbar_fence_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  bool ok = true;
  auto wait = [&](uint64_t* m, int parity) { if (ok) ok = tc::mbar_wait(m, (uint32_t)parity & 1u); };
  auto arrive = [&](uint64_t* m) {  // of a whole warp
    __syncwarp();
    if (lane == 0) mbar_arrive(m);
  };
  auto stage = [&](int it) { return sm + (it & 1) * kScanStage; };
  auto fresh = [](tc::Tile t) {  // keeps the descriptors of a product from being held in registers from chunk to chunk
    asm volatile("" : "+r"(t.saddr));
    return t;
  };

  if (warp < 4) {  // ---- the state: thread = row, all 64 columns
    tc::reg_inc<104>();
    f2 H[P / 2];
#pragma unroll
    for (int x = 0; x < P / 2; ++x) H[x] = 0ull;
    for (int it = 0; it < n; ++it) {
      const int a = it & 1;
      if (it > 0) wait(hfree, it - 1);
#pragma unroll
      for (int x = 0; x < P / 8; ++x)
        sts16(Ht, tc::kmajor_unit(tid, x, P), make_uint4(narrow2(H[4 * x]), narrow2(H[4 * x + 1]), narrow2(H[4 * x + 2]), narrow2(H[4 * x + 3])));
      tc::fence_async_smem();
      arrive(hready);
      wait(full + a, it >> 1);
      wait(accfull + a, it >> 1);
      tc::fence_after_sync();
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        const f2 L = dup2(scal[a].L);
#pragma unroll
        for (int q = 0; q < P; q += 8) {
          f2 f[4];
          ld_pairs(taddr + 64 * a + q, warp, f);
          tc::tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 4; ++x) H[q / 2 + x] = mad2(L, H[q / 2 + x], f[x]);
        }
      }
      tc::fence_before_sync();
      arrive(accfree + a);
      arrive(sfree + a);
    }
  } else if (warp < 8) {  // ---- G*M and y: this thread's row and the half of the columns that it holds of every result
    tc::reg_inc<72>();
    const int t = 32 * (warp & 1) + lane, n0 = 32 * ((warp >> 1) & 1);
    for (int it = 0; it < n; ++it) {
      const ChunkScal& s = scal[it & 1];
      uint8_t* S = stage(it);
      wait(full + (it & 1), it >> 1);
      wait(accfull + (it & 1), it >> 1);  // (Brot makes room)
      wait(gfull, it);
      tc::fence_after_sync();
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        float f[32];
        ld_acc32(taddr + tG, warp, 0, f);
        mask_row(f, s, t, n0);
#pragma unroll
        for (int x = 0; x < 4; ++x) sts16(S, tc::kmajor_unit(t, (n0 >> 3) + x, Q), pack8(&f[8 * x]));
      }
      tc::fence_before_sync();
      tc::fence_async_smem();
      arrive(gmready);
      wait(yfull, it);
      tc::fence_after_sync();
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {  // y = (G*M) X + exp(Lam) Crot H0
        const float de = s.dexp[t];
#pragma unroll
        for (int q = 0; q < 32; q += 16) {
          float f[16], h[16];
          ld_acc16(taddr + tY, warp, q, f);
          ld_acc16(taddr + tH, warp, q, h);
#pragma unroll
          for (int x = 0; x < 16; ++x) f[x] = fmaf(de, h[x], f[x]);
          sts16(S + 32768, tc::sw128_unit(t, (n0 + q) >> 3), pack8(f));
          sts16(S + 32768, tc::sw128_unit(t, ((n0 + q) >> 3) + 1), pack8(f + 8));
        }
      }
      tc::fence_before_sync();
      arrive(yfree);
      tc::fence_async_smem();
      arrive(yready + (it & 1));
    }
  } else if (warp < 12) {  // ---- rows rotated, x scaled
    tc::reg_dec<48>();
    const int u0 = tid - 256;
    for (int it = 0; it < n; ++it) {
      const ChunkScal& s = scal[it & 1];
      uint8_t* S = stage(it);
      wait(full + (it & 1), it >> 1);
      rotate_in_tile<true>(S, s.sn, s.cs, u0, 128);
      if (it > 0) wait(xsfree, it - 1);
      scale_rows(Xs, S + 32768, s.re, u0, 128);
      tc::fence_async_smem();
      arrive(readyb + (it & 1));
      rotate_in_tile<true>(S + 16384, s.sn, s.cs, u0, 128);
      tc::fence_async_smem();
      arrive(readyc + (it & 1));
    }
  } else {
    tc::reg_dec<32>();
    if (warp == 12) {  // ---- copies
      if (lane == 0) {
        int issued = 0;
        for (int it = 0; it < n; ++it) {
          const int s = it & 1;
          uint8_t* S = stage(it);
          if (it > 1) wait(sfree + s, (it >> 1) - 1);
          if (!ok) break;
          ++issued;
          tc::mbar_expect_tx(full + s, (uint32_t)kScanStage + (uint32_t)sizeof(ChunkScal));
          for (int sl = 0; sl < 2; ++sl) tc::tma_load_4d(tc::smem_u32(S) + 8192 * sl, &maps.b, 64 * sl, g, it * Q, b, full + s);
          tc::tma_load_4d(tc::smem_u32(S) + 32768, &maps.x, 0, head, it * Q, b, full + s);
          tc::bulk_load(tc::smem_u32(scal + s), p.cs + (cbase + it) * (sizeof(ChunkScal) / 4), (uint32_t)sizeof(ChunkScal), full + s);
          for (int sl = 0; sl < 2; ++sl) tc::tma_load_4d(tc::smem_u32(S) + 16384 + 8192 * sl, &maps.c, 64 * sl, g, it * Q, b, full + s);
        }
        for (int q = max(0, issued - 2); q < issued; ++q) tc::mbar_wait(full + (q & 1), (q >> 1) & 1);  // (outlive the copies)
      }
    } else if (warp == 13) {  // ---- products of the state
      if (tc::elect_one()) {
        for (int it = 0; it < n; ++it) {
          const int a = it & 1;
          wait(readyb + a, it >> 1);
          if (it > 1) wait(accfree + a, (it >> 1) - 1);
          if (!ok) break;
          tc::fence_after_sync();
          // [128 n x 64 p] = Brot^T diag(r e) X, both contracted over their rows
          tc::issue_gemm(taddr + 64 * a, fresh(tc::mnmajor_sw128_tile(stage(it), 8192)), fresh(tc::mnmajor_sw128_tile(Xs, 8192)), 128, P, Q, false);
          tc::mma_commit(accfull + a);
          tc::mma_commit(xsfree);
        }
      }
    } else if (warp == 14) {  // ---- products of the output
      if (tc::elect_one()) {
        for (int it = 0; it < n; ++it) {
          wait(readyb + (it & 1), it >> 1);
          wait(readyc + (it & 1), it >> 1);
          if (!ok) break;
          tc::fence_after_sync();
          tc::issue_gemm<true>(taddr + tG, fresh(tc::kmajor_sw128_tile(stage(it) + 16384, 8192)), fresh(tc::kmajor_sw128_tile(stage(it), 8192)), 64, Q, N, false);  // G = Crot Brot^T
          tc::mma_commit(gfull);
          wait(hready, it);
          if (it > 0) wait(yfree, it - 1);
          if (!ok) break;
          tc::fence_after_sync();
          tc::issue_gemm<true>(taddr + tH, fresh(tc::kmajor_sw128_tile(stage(it) + 16384, 8192)), fresh(tc::mnmajor_tile(Ht, P)), 64, P, N, false);         // Crot H0
          tc::mma_commit(hfree);
          wait(gmready, it);
          if (!ok) break;
          tc::fence_after_sync();
          tc::issue_gemm<true>(taddr + tY, fresh(tc::kmajor_tile(stage(it), Q)), fresh(tc::mnmajor_sw128_tile(stage(it) + 32768, 8192)), 64, P, Q, false);  // (G*M) X
          tc::mma_commit(yfull);
        }
      }
    } else {  // ---- stores
      if (lane == 0) {
        for (int it = 0; it < n; ++it) {
          uint8_t* S = stage(it);
          wait(hready, it);
          if (!ok) break;
          if (save) {
            tc::bulk_store(p.H0 + (cbase + it) * (N * P), tc::smem_u32(Ht), 16384);
            tc::bulk_commit();
            tc::bulk_wait_read<0>();
          }
          mbar_arrive(hfree);
          wait(yready + (it & 1), it >> 1);
          if (!ok) break;
          tc::tma_store_4d(&maps.y, tc::smem_u32(S) + 32768, 0, head, it * Q, b);
          tc::bulk_commit();
          tc::bulk_wait_read<0>();
          mbar_arrive(sfree + (it & 1));
        }
      }
    }
    __syncwarp();
    ok = __all_sync(0xffffffffu, ok);
  }
  if (!ok && lane == 0) atomicExch(p.status, 14);
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 256);
}

// ------------------------------------------------------------ chunk gradients
// One CTA per chunk and up to kGradHeads heads of a group.  The heads of a group share B and C and differ by one angle per
// step, so nothing is rotated: with J(e, o) = (-o, e) on every pair of states and delta = phi_t - phi_s
//     Crot_t . Brot_s = cos(delta) (C B^T)_ts + sin(delta) (C (J B)^T)_ts
//     (Crot H0)_t     = cos(phi_t) (C H0)_t + sin(phi_t) (CJ H0)_t,   CJ = J^T C
// the two 64 x 64 products stay in registers for all heads, and what the heads add to dB and dC is summed before it meets
// B and C: over the 64 x 64 products in registers (W1, W2), over the chunk states in tensor memory,
//     dC = W1 B + W2 (J B) + Z1 + J Z2,   Z1 = sum_h (cos e^Lam dY) H0^T,  Z2 = sum_h (sin e^Lam dY) H0^T
//     dB = W1^T C + W2^T CJ + Y1 + J Y2,  Y1 = sum_h (cos r e x) dH1^T,     Y2 = sum_h (sin r e x) dH1^T
//     W1_ts = sum_h cos(delta) dG_ts,  W2_ts = sum_h sin(delta) dG_ts,      dG = (dY X^T) * M
// so one partial image of dB and dC leaves per CTA instead of one per head.  W1 and W2 are operands of products, so they are
// rounded to bf16, once, after the sum over the heads.
//
// One CTA per SM: 16 warps with a row t and 8 of 64 columns of every product, one warp that issues the copies, one that
// issues the products (an elected thread of a warp of its own: 33 cycles an instruction, 60 behind a test of the thread's
// index), one that finishes the per-step scalars and one that stores dx; everything is handed over by mbarriers.
// Products of a head: dP = dY X^T, U = {C, CJ} H0, V = {B, JB} dH1 (asked for a head ahead), Z and Y, then dX = (G*M)^T dY.
// 8 x 4096 x 32 heads: 335 us + 29 for the row sums behind it, 1.0 GB (0.15 ms); a CTA per head and chunk that rotated B and C
// took 527 + 118 with 1.5 + 0.6 GB.  Bound by instruction issue: most of a head is the arithmetic of the 64 x 64 products, of U
// and V and of the scaled images at half of the issue slots; pairs of columns in packed registers (7.8 k cycles a head without,
// 5.0 k with them, 4.7 k since U and V meet x and dY as they landed instead of two images each: also the closer result, the
// images are rounded to bf16: dtheta 8.1e-4 -> 7.0e-4 from float64, ddt 5.9e-4 -> 5.4e-4).
// TMEM: Z [0,128), Y [128,256), U [256,320), V [320,384), dP [384,416), dX [416,448); at the start C B^T and C (J B)^T in
// the last two, at the end the products with W1 and W2 in U and V.
constexpr int kGradWarps = 16;
constexpr int kGradThreads = 32 * (kGradWarps + 4);
constexpr int kGradStage = 2 * 8192 + 2 * 16384;  // x, dY, H0, dH1 of a head
constexpr int kGradPart = (8 * 4 * Q + 5 * Q + 32) * 4;
constexpr int kGradSmem = 4 * 16384 + 2 * kGradStage + 4 * 8192 + 8192 + 8192 + kGradPart + 4 * (int)sizeof(ChunkScal) + 24 * 8 + 16 + 1024;
static_assert(kGradSmem <= 227 * 1024, "one CTA per SM");
constexpr int kGradPitch = N + 4;  // floats per row of the sums on their way out (over the stages)
static_assert(2 * Q * kGradPitch * 4 <= 2 * kGradStage, "two tiles of row sums fit into the stages");

template <bool TMA>
__global__ void __launch_bounds__(kGradThreads, 1) m3s_chunk_grad_kernel(SsdP p, const __grid_constant__ ChunkMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Bt = sm;                    // [64][128] B, J B, C, CJ (swizzled slabs)
  uint8_t* Jt = Bt + 16384;
  uint8_t* Ct = Jt + 16384;
  uint8_t* Kt = Ct + 16384;
  uint8_t* Yc = Kt + 16384;            // [64][64] cos e^Lam dY, then sin e^Lam dY, cos r e x, sin r e x (swizzled like their sources)
  uint8_t* Xc = Yc + 2 * 8192;
  uint8_t* GMt = Xc + 2 * 8192;        // [64][64] G*M
  uint8_t* Dx = GMt + 8192;            // [64][64] dx on its way out (swizzled)
  uint8_t* St = Dx + 8192;             // two stages: x, dY (swizzled), H0, dH1 (images)
  ChunkScal* scal = reinterpret_cast<ChunkScal*>(St + 2 * kGradStage);  // x4: the scalars of a head (read longer than its tiles)
  float* part = reinterpret_cast<float*>(scal + 4);  // [8 column groups][4][Q]: dLam, de, dphi (negative: by the states read), dphi row partials
  float* csw = part + 8 * 4 * Q;       // [2][2][Q] column sums over the two halves of the rows: of dM*D (s < t), of dG dG/ddelta
  float* dgs = csw + 4 * Q;            // [Q] dgam
  float* red = dgs + Q;                // [16] <dH1, H0>, [16] <dH1, J H0> per warp
  uint64_t* full = reinterpret_cast<uint64_t*>(red + 32);  // x2: a head's operands landed
  uint64_t* freed = full + 2;          // x2: and are no longer needed
  uint64_t* tiles = freed + 2;         // B, C landed
  uint64_t* images = tiles + 1;        // the scaled images of a head are written (first: J B and CJ; last: W1 and W2)
  uint64_t* gready = images + 1;       // G*M is written
  uint64_t* uvfree = gready + 1;       // dP, U, V are read
  uint64_t* pready = uvfree + 1;       // row partials are written
  uint64_t* pfree = pready + 1;
  uint64_t* xready = pfree + 1;        // dx is written
  uint64_t* xfree = xready + 1;
  uint64_t* m1 = xfree + 1;            // products: dP, U, V
  uint64_t* m2 = m1 + 1;               // products: Z, Y, dX
  uint64_t* m0 = m2 + 1;               // products of the start
  uint32_t* tslot = reinterpret_cast<uint32_t*>(m0 + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x, b = blockIdx.z, t0 = c * Q;
  const int per = p.NH / p.G, g = blockIdx.y / p.splits, sp = blockIdx.y % p.splits;
  const int h0 = g * per + sp * p.hp, nh = min(p.hp, g * per + per - h0);  // this CTA's heads
  auto unit_of = [&](int head) { return ((size_t)b * p.NH + head) * p.n + c; };

  if (warp == 0) { tc::tmem_alloc(tslot, 512); tc::tmem_relinquish(); }
  if (tid == 32) {
    for (int s = 0; s < 2; ++s) {
      tc::mbar_init(full + s, TMA ? 1 : 33); tc::mbar_init(freed + s, kGradWarps + 1);
    }
    tc::mbar_init(tiles, TMA ? 1 : 32);
    tc::mbar_init(images, kGradWarps); tc::mbar_init(gready, kGradWarps); tc::mbar_init(uvfree, kGradWarps);
    tc::mbar_init(pready, kGradWarps); tc::mbar_init(pfree, 1); tc::mbar_init(xready, kGradWarps); tc::mbar_init(xfree, 1);
    tc::mbar_init(m0, 1); tc::mbar_init(m1, 1); tc::mbar_init(m2, 1);
    tc::mbar_fence_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  bool ok = true;
  auto wait = [&](uint64_t* m, int parity) { if (ok) ok = tc::mbar_wait(m, (uint32_t)parity & 1u); };
  auto arrive = [&](uint64_t* m) {  // of a whole warp
    __syncwarp();
    if (lane == 0) mbar_arrive(m);
  };
  constexpr uint32_t tZ = 0, tY = 128, tU = 256, tV = 320, tP = 384, tX = 416;

  if (warp == kGradWarps) {  // ---- copies
    tc::reg_dec<40>();
    if (TMA) {
      if (lane == 0) {
        tc::mbar_expect_tx(tiles, 2 * 16384);
        for (int sl = 0; sl < 2; ++sl) {
          tc::tma_load_4d(tc::smem_u32(Bt) + 8192 * sl, &maps.b, 64 * sl, g, t0, b, tiles);
          tc::tma_load_4d(tc::smem_u32(Ct) + 8192 * sl, &maps.c, 64 * sl, g, t0, b, tiles);
        }
      }
    } else {
      const size_t row = ((size_t)b * p.T + t0) * p.G + g;
      for (int sl = 0; sl < 2; ++sl) {
        stage_slab(tc::smem_u32(Bt) + 8192 * sl, p.b + row * N + 64 * sl, p.T, (size_t)p.G * N, t0, lane, 32);
        stage_slab(tc::smem_u32(Ct) + 8192 * sl, p.c + row * N + 64 * sl, p.T, (size_t)p.G * N, t0, lane, 32);
      }
      tc::cp_async_wait_all();
      tc::fence_async_smem();
      mbar_arrive(tiles);
    }
    int issued = 0;
    for (int h = 0; h < nh; ++h) {
      const int s = h & 1, head = h0 + h;
      if (h > 1) wait(freed + s, (h >> 1) - 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      uint8_t* S = St + s * kGradStage;
      if (lane == 0) {
        tc::mbar_expect_tx(full + s, (uint32_t)kGradStage + (uint32_t)sizeof(ChunkScal) - (TMA ? 0u : 16384u));
        if (TMA) {
          tc::tma_load_4d(tc::smem_u32(S), &maps.x, 0, head, t0, b, full + s);
          tc::tma_load_4d(tc::smem_u32(S) + 8192, &maps.dy, 0, head, t0, b, full + s);
        }
        tc::bulk_load(tc::smem_u32(S) + 16384, p.H0 + unit_of(head) * (N * P), 16384, full + s);
        tc::bulk_load(tc::smem_u32(S) + 32768, p.dH1 + unit_of(head) * (N * P), 16384, full + s);
        tc::bulk_load(tc::smem_u32(scal + (h & 3)), p.cs + unit_of(head) * (sizeof(ChunkScal) / 4), (uint32_t)sizeof(ChunkScal), full + s);
      }
      ++issued;
      if (!TMA) {
        const size_t row = (size_t)b * p.T + t0;
        stage_slab(tc::smem_u32(S), p.x + row * p.D + head * P, p.T, p.D, t0, lane, 32);
        stage_slab(tc::smem_u32(S) + 8192, p.dy + row * p.D + head * P, p.T, p.D, t0, lane, 32);
        tc::cp_async_wait_all();
        tc::fence_async_smem();
        mbar_arrive(full + s);
      }
    }
    for (int q = max(0, issued - 2); q < issued; ++q) tc::mbar_wait(full + (q & 1), (q >> 1) & 1);  // (outlive the copies)
  } else if (warp == kGradWarps + 1) {  // ---- products
    tc::reg_dec<40>();
    if (tc::elect_one()) {
      wait(images, 0);
      tc::fence_after_sync();
      if (ok) {
        tc::issue_gemm<true>(taddr + tP, tc::kmajor_sw128_tile(Ct, 8192), tc::kmajor_sw128_tile(Bt, 8192), 64, Q, N, false);
        tc::issue_gemm<true>(taddr + tX, tc::kmajor_sw128_tile(Kt, 8192), tc::kmajor_sw128_tile(Bt, 8192), 64, Q, N, false);
        tc::mma_commit(m0);
      }
      for (int h = 0; h < nh && ok; ++h) {
        const int s = h & 1;
        uint8_t* S = St + s * kGradStage;
        wait(full + s, h >> 1);
        wait(uvfree, h);  // (once more at the start: the first products have been read)
        tc::fence_after_sync();
        if (!ok) break;
        const tc::Tile X = tc::kmajor_sw128_tile(S, 8192), Y = tc::kmajor_sw128_tile(S + 8192, 8192);
        const tc::Tile H = tc::mnmajor_tile(S + 16384, P), D = tc::mnmajor_tile(S + 32768, P);
        tc::issue_gemm<true>(taddr + tP, Y, X, 64, Q, P, false);
        tc::issue_gemm<true>(taddr + tU, tc::kmajor_sw128_tile(Ct, 8192), H, 64, P, N, false);
        tc::issue_gemm<true>(taddr + tU + 32, tc::kmajor_sw128_tile(Kt, 8192), H, 64, P, N, false);
        tc::issue_gemm<true>(taddr + tV, tc::kmajor_sw128_tile(Bt, 8192), D, 64, P, N, false);
        tc::issue_gemm<true>(taddr + tV + 32, tc::kmajor_sw128_tile(Jt, 8192), D, 64, P, N, false);
        tc::mma_commit(m1);
        wait(images, h + 1);
        tc::fence_after_sync();
        if (!ok) break;
        tc::issue_gemm(taddr + tZ, tc::kmajor_sw128_tile(Yc, 8192), tc::kmajor_tile(S + 16384, P), 128, N, P, h > 0);
        tc::issue_gemm(taddr + tY, tc::kmajor_sw128_tile(Xc, 8192), tc::kmajor_tile(S + 32768, P), 128, N, P, h > 0);
        wait(gready, h);
        tc::fence_after_sync();
        if (!ok) break;
        tc::issue_gemm<true>(taddr + tX, tc::mnmajor_tile(GMt, Q), tc::mnmajor_sw128_tile(S + 8192, 8192), 64, P, Q, false);
        tc::mma_commit(m2);
        tc::mma_commit(freed + s);
      }
      wait(images, nh + 1);
      wait(uvfree, nh);
      tc::fence_after_sync();
      if (ok) {  // W1, W2 (images over the scaled ones)
        tc::issue_gemm<true>(taddr + tU, tc::kmajor_tile(Yc, Q), tc::mnmajor_sw128_tile(Bt, 8192), 64, N, Q, false);
        tc::issue_gemm<true>(taddr + tU, tc::kmajor_tile(Yc + 8192, Q), tc::mnmajor_sw128_tile(Jt, 8192), 64, N, Q, true);
        tc::issue_gemm<true>(taddr + tV, tc::mnmajor_tile(Yc, Q), tc::mnmajor_sw128_tile(Ct, 8192), 64, N, Q, false);
        tc::issue_gemm<true>(taddr + tV, tc::mnmajor_tile(Yc + 8192, Q), tc::mnmajor_sw128_tile(Kt, 8192), 64, N, Q, true);
        tc::mma_commit(m1);
      }
    }
    __syncwarp();
  } else if (warp == kGradWarps + 2) {  // ---- per-step scalars
    tc::reg_dec<40>();
    for (int h = 0; h < nh; ++h) {
      const ChunkScal& s = scal[h & 3];
      wait(pready, h);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      auto part_sum = [&](int what, int q) {
        float v[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) v[x] = part[(4 * x + what) * Q + q];
        return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
      };
      const int ra = Q - 1 - 2 * lane, rb = ra - 1;
      const float zra = part_sum(1, ra), zrb = part_sum(1, rb);            // r_s zeta_s
      const float cea = csw[ra] + csw[Q + ra], ceb = csw[rb] + csw[Q + rb];
      const float dga = dgs[ra], dgb = dgs[rb], bsa = part_sum(2, ra), bsb = part_sum(2, rb);
      // (the angle in double precision: steps whose gradient is small stand behind sums over large ones that cancel)
      double dpa = (double)part_sum(3, ra) - bsa - (csw[2 * Q + ra] + csw[3 * Q + ra]);
      double dpb = (double)part_sum(3, rb) - bsb - (csw[2 * Q + rb] + csw[3 * Q + rb]);
      const float dla = part_sum(0, ra), dlb = part_sum(0, rb);
      const float hw = red[lane];
      const float ea = s.e[ra], eb = s.e[rb], ga = s.gam[ra], gb = s.gam[rb], L = s.L;
      arrive(pfree);
      const float hh = warp_sum(lane < kGradWarps ? hw : 0.f);
      const double later = warp_sum((lane < kGradWarps ? 0.0 : (double)L * hw) + ((double)bsa + bsb));
      const float zs = warp_sum(fmaf(ea, zra, eb * zrb));
      const float base = zs + L * hh;  // d/dLam_end
      // dLam -> da: reverse in-chunk cumulative sum
      float a = dla - ea * zra - (ea * cea + ga * dga);
      float bq = dlb - eb * zrb - (eb * ceb + gb * dgb);
      warp_rcumsum64(a, bq, lane);
      // and dphi -> the sum over this and all later steps, which is what theta and dt get: later steps enter through the states
      // at the end of the chunk (summed up step by step, the error of the rounded states grew with the length of the sequence)
      warp_rcumsum64(dpa, dpb, lane);
      dpa += later;
      dpb += later;
      const size_t o = ((size_t)b * p.NH + h0 + h) * p.T + t0;
      if (t0 + ra < p.T) { p.da[o + ra] = base + a; p.de[o + ra] = zra + cea; p.dgam[o + ra] = dga; p.dphi[o + ra] = (float)dpa; }
      if (t0 + rb < p.T) { p.da[o + rb] = base + bq; p.de[o + rb] = zrb + ceb; p.dgam[o + rb] = dgb; p.dphi[o + rb] = (float)dpb; }
    }
  } else if (warp == kGradWarps + 3) {  // ---- dx
    tc::reg_dec<40>();
    for (int h = 0; h < nh; ++h) {
      wait(xready, h);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (TMA) {
        if (lane == 0) {
          tc::tma_store_4d(&maps.dx, tc::smem_u32(Dx), 0, h0 + h, t0, b);
          tc::bulk_commit();
          tc::bulk_wait_read<0>();
        }
      } else {
        for (int u = lane; u < Q * 8; u += 32) {
          const int t = u >> 3, c8 = u & 7;
          if (t0 + t < p.T)
            *reinterpret_cast<uint4*>(p.dx + ((size_t)b * p.T + t0 + t) * p.D + (h0 + h) * P + 8 * c8) =
                *reinterpret_cast<const uint4*>(Dx + t * 128 + ((c8 ^ (t & 7)) << 4));
        }
      }
      arrive(xfree);
    }
  } else if (warp < kGradWarps) {  // ---- rows and columns
    tc::reg_inc<104>();  // (16 x 104 + 4 x 40 registers a lane, of 20 x 96 at launch)
    // this thread's row, its 8 of 64 columns of a result and their first TMEM column
    const int t = 32 * (warp & 1) + lane, tc8 = 8 * (warp >> 2), n8 = 32 * ((warp >> 1) & 1) + tc8, slot = 4 * ((warp >> 1) & 1) + (warp >> 2);
    wait(tiles, 0);
    for (int u = tid; u < Q * 16; u += 32 * kGradWarps) {  // J B = (-o, e), CJ = (o, -e) of every pair
      const uint4 vb = *reinterpret_cast<const uint4*>(Bt + 16 * u), vc = *reinterpret_cast<const uint4*>(Ct + 16 * u);
      auto sw = [](uint32_t x, uint32_t sign) { return __byte_perm(x, x, 0x1032) ^ sign; };
      *reinterpret_cast<uint4*>(Jt + 16 * u) = make_uint4(sw(vb.x, 0x8000u), sw(vb.y, 0x8000u), sw(vb.z, 0x8000u), sw(vb.w, 0x8000u));
      *reinterpret_cast<uint4*>(Kt + 16 * u) =
          make_uint4(sw(vc.x, 0x80000000u), sw(vc.y, 0x80000000u), sw(vc.z, 0x80000000u), sw(vc.w, 0x80000000u));
    }
    tc::fence_async_smem();
    arrive(images);
    wait(m0, 0);
    tc::fence_after_sync();
    f2 g1[4] = {}, g2[4] = {}, w1[4] = {}, w2[4] = {};  // C B^T, C (J B)^T; the sums over the heads
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      ld_pairs(taddr + tP + tc8, warp, g1);
      ld_pairs(taddr + tX + tc8, warp, g2);
      tc::tmem_ld_wait();
#pragma unroll
      for (int x = 0; x < 4; ++x) {  // (causal part only)
        const float2 a = unpack2(g1[x]), d = unpack2(g2[x]);
        const bool in0 = n8 + 2 * x <= t, in1 = n8 + 2 * x + 1 <= t;
        g1[x] = pack2(in0 ? a.x : 0.f, in1 ? a.y : 0.f);
        g2[x] = pack2(in0 ? d.x : 0.f, in1 ? d.y : 0.f);
      }
    }
    tc::fence_before_sync();
    arrive(uvfree);
    const bool above = n8 > t - lane + 31;               // the warp's rows lie wholly above these columns
    const bool diagonal = (n8 >> 5) == (warp & 1);        // its rows and columns may meet
    const uint32_t tunit = (uint32_t)t * 128u + (uint32_t)(((n8 >> 3) ^ (t & 7)) << 4);  // this thread's 16 bytes of a swizzled tile
    for (int h = 0; h < nh; ++h) {
      uint8_t* S = St + (h & 1) * kGradStage;
      const ChunkScal& s = scal[h & 3];
      wait(full + (h & 1), h >> 1);
      {  // scaled images: one unit of x and of dY per thread (unit u lies in row u / 8)
        const int r = tid >> 3;
        const float sn = s.sn[r], cs = s.cs[r], xd = s.dexp[r], xr = s.re[r];
        auto put = [&](const uint8_t* src, uint8_t* dst, float sc, float ss) {
          const uint4 x = *reinterpret_cast<const uint4*>(src + 16 * tid);
          const f2 v[4] = {widen2(x.x), widen2(x.y), widen2(x.z), widen2(x.w)}, c2 = dup2(sc), s2 = dup2(ss);
          *reinterpret_cast<uint4*>(dst + 16 * tid) =
              make_uint4(narrow2(mul2(v[0], c2)), narrow2(mul2(v[1], c2)), narrow2(mul2(v[2], c2)), narrow2(mul2(v[3], c2)));
          *reinterpret_cast<uint4*>(dst + 8192 + 16 * tid) =
              make_uint4(narrow2(mul2(v[0], s2)), narrow2(mul2(v[1], s2)), narrow2(mul2(v[2], s2)), narrow2(mul2(v[3], s2)));
        };
        put(S + 8192, Yc, xd * cs, xd * sn);
        put(S, Xc, xr * cs, xr * sn);
      }
      tc::fence_async_smem();
      arrive(images);
      float hh = 0.f, jj = 0.f;  // <dH1, H0> and <dH1, J H0>
      // By the warps that have nothing below the diagonal in the product to come: blocks of 16 state rows of dH1 times the
      // same rows of H0 (mma.sync), whose diagonals and their neighbours are the row products that are wanted.
      if (above) {
        const uint32_t sh = tc::smem_u32(S + 16384), sd = sh + 16384;
        float d1[4] = {}, d2[4] = {};
#pragma unroll
        for (int blk = 0; blk < 2; ++blk)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint32_t u = tc::kmajor_unit(32 * (warp >> 2) + 16 * blk + (lane & 15), 2 * ks + (lane >> 4), P);
            uint32_t a[4], o[4];
            ms::ldsm(a, sd + u);
            ms::ldsm(o, sh + u);
            ms::mma(d1, a, o[0], o[2]);  // rows 0-7 of H0: wanted in rows 0-7 of the block
            ms::mma(d2, a, o[1], o[3]);  // rows 8-15
          }
        // (sums over both blocks) this lane has row lane / 4 and columns 2 (lane % 4), + 1
        if ((lane >> 3) == (lane & 3)) {
          const bool odd = (lane >> 2) & 1;
          hh = odd ? d1[1] + d2[3] : d1[0] + d2[2];
          jj = odd ? d1[0] + d2[2] : -(d1[1] + d2[3]);
        }
      }
      wait(m1, h);
      tc::fence_after_sync();
      ok = __all_sync(0xffffffffu, ok);
      const float lt = s.Lam[t], gt = s.gam[t], ct = s.cs[t], st = s.sn[t];
      float dg = 0.f;
      f2 dl = 0, dphi = 0, pya = 0, pyb = 0, pxa = 0;  // row sums; of dY with C H0 and CJ H0, of x with B dH1 (and (J B) dH1)
      float ce[8] = {}, cq[8] = {};
      if (ok) {
        uint32_t gm[4] = {};
        if (!above) {
          f2 fd[4];
          ld_pairs(taddr + tP + tc8, warp, fd);
          tc::tmem_ld_wait();
          const f2 lt2 = dup2(lt), ct2 = dup2(ct), st2 = dup2(st), nct2 = dup2(-ct), one = dup2(-1.f), log2e = dup2(1.4426950408889634f);
          const int k = t - n8;
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const ulonglong2 l4 = *reinterpret_cast<const ulonglong2*>(s.Lam + n8 + 4 * x), e4 = *reinterpret_cast<const ulonglong2*>(s.e + n8 + 4 * x);
            const ulonglong2 c4 = *reinterpret_cast<const ulonglong2*>(s.cs + n8 + 4 * x), s4 = *reinterpret_cast<const ulonglong2*>(s.sn + n8 + 4 * x);
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              const int z = 2 * x + y, q = 2 * z;
              const f2 cc = y ? c4.y : c4.x, ss = y ? s4.y : s4.x;
              const float2 arg = unpack2(mul2(mad2(y ? l4.y : l4.x, one, lt2), log2e)), es = unpack2(y ? e4.y : e4.x), pd = unpack2(fd[z]);
              // selects, no branches: the exponentials of different columns overlap
              const f2 D = pack2(q <= k ? ex2(arg.x) : 0.f, q + 1 <= k ? ex2(arg.y) : 0.f);
              const f2 M = mul2(D, pack2(q < k ? es.x : gt, q + 1 < k ? es.y : gt));
              const f2 dP = pack2(q <= k ? pd.x : 0.f, q + 1 <= k ? pd.y : 0.f);
              const f2 cd = mad2(ct2, cc, mul2(st2, ss)), sd = mad2(st2, cc, mul2(nct2, ss));
              const f2 gv = mad2(cd, g1[z], mul2(sd, g2[z])), gd = mad2(mul2(sd, g1[z]), one, mul2(cd, g2[z]));  // G, dG/ddelta
              const f2 dG = mul2(dP, M), dM = mul2(dP, gv), dw = mul2(dM, D), qq = mul2(dG, gd);
              gm[z] = narrow2(mul2(gv, M));
              fma2(dl, dM, M);
              dphi = add2(dphi, qq);            // row sums minus column sums
              fma2(w1[z], dG, cd);
              fma2(w2[z], dG, sd);
              const float2 q2 = unpack2(qq), w = unpack2(dw);
              cq[q] = q2.x; cq[q + 1] = q2.y;
              ce[q] = w.x; ce[q + 1] = w.y;     // de_s: column sums, without the diagonal
            }
          }
          if (diagonal) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              dg = q == k ? ce[q] : dg;
              ce[q] = q < k ? ce[q] : 0.f;
            }
          }
        }
        sts16(GMt, tc::kmajor_unit(t, n8 >> 3, Q), make_uint4(gm[0], gm[1], gm[2], gm[3]));
      }
      tc::fence_async_smem();
      arrive(gready);
      // U, V: kappa_t = e^Lam dY_t . (Crot H0)_t, zeta_s = x_s . (Brot dH1)_s and their derivatives by the angle.  dY and x as they
      // landed: the factors of a row are applied to its sums.
      f2 v[4] = {}, pxb = 0;
      if (ok) {
        f2 fa[4], fb[4];
        auto word = [](const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; };
        ld_pairs(taddr + tU + tc8, warp, fa);
        ld_pairs(taddr + tU + 32 + tc8, warp, fb);
        const uint4 iy = *reinterpret_cast<const uint4*>(S + 8192 + tunit);
        tc::tmem_ld_wait();
#pragma unroll
        for (int z = 0; z < 4; ++z) {
          const f2 y = widen2(word(iy, z));
          fma2(pya, y, fa[z]);
          fma2(pyb, y, fb[z]);
        }
        ld_pairs(taddr + tV + tc8, warp, fa);
        ld_pairs(taddr + tV + 32 + tc8, warp, fb);
        const uint4 ix = *reinterpret_cast<const uint4*>(S + tunit);
        const f2 ct2 = dup2(ct), nst2 = dup2(-st);
        tc::tmem_ld_wait();
#pragma unroll
        for (int z = 0; z < 4; ++z) {
          const f2 xz = widen2(word(ix, z));
          fma2(pxa, xz, fa[z]);
          fma2(pxb, xz, fb[z]);
          v[z] = mad2(ct2, fa[z], mul2(nst2, fb[z]));   // Brot = cos B - sin (J B)
        }
      }
      tc::fence_before_sync();
      arrive(uvfree);
      colsum8(ce, lane);
      colsum8(cq, lane);
      const float acc = above ? warp_sum(hh) : 0.f, accj = above ? warp_sum(jj) : 0.f;
      if (h > 0) wait(pfree, h - 1);
      if (lane < 8) {
        csw[(warp & 1) * Q + n8 + lane] = ce[0];
        csw[(2 + (warp & 1)) * Q + n8 + lane] = cq[0];
      }
      const float ret = s.re[t], det = s.dexp[t], ya = sum2(pya), yb = sum2(pyb), xa = sum2(pxa), xb = sum2(pxb);
      part[(4 * slot + 0) * Q + t] = fmaf(det, fmaf(ct, ya, st * yb), sum2(dl));
      part[(4 * slot + 1) * Q + t] = s.r[t] * fmaf(ct, xa, -(st * xb));
      part[(4 * slot + 2) * Q + t] = ret * fmaf(ct, xb, st * xa);
      if ((t >> 3) == (n8 >> 3)) dgs[t] = dg;
      part[(4 * slot + 3) * Q + t] = fmaf(det, fmaf(ct, yb, -(st * ya)), sum2(dphi));
      if (lane == 0) {
        red[warp] = acc;
        red[kGradWarps + warp] = accj;
      }
      arrive(pready);
      wait(m2, h);
      tc::fence_after_sync();
      if (h > 0) wait(xfree, h - 1);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {  // dx_s = (G*M)^T dY + r e (Brot dH1)
        f2 f[4];
        ld_pairs(taddr + tX + tc8, warp, f);
        tc::tmem_ld_wait();
        const f2 r2 = dup2(ret);
        *reinterpret_cast<uint4*>(Dx + tunit) = make_uint4(narrow2(mad2(r2, v[0], f[0])), narrow2(mad2(r2, v[1], f[1])),
                                                           narrow2(mad2(r2, v[2], f[2])), narrow2(mad2(r2, v[3], f[3])));
      }
      tc::fence_before_sync();
      tc::fence_async_smem();
      arrive(xready);
      arrive(freed + (h & 1));
    }
    // the sums over the heads
    sts16(Yc, tc::kmajor_unit(t, n8 >> 3, Q), make_uint4(narrow2(w1[0]), narrow2(w1[1]), narrow2(w1[2]), narrow2(w1[3])));
    sts16(Yc + 8192, tc::kmajor_unit(t, n8 >> 3, Q), make_uint4(narrow2(w2[0]), narrow2(w2[1]), narrow2(w2[2]), narrow2(w2[3])));
    tc::fence_async_smem();
    tc::fence_before_sync();
    arrive(images);
    // while they meet B and C: the sums over the chunk states, put together over the stages
    float* Sum = reinterpret_cast<float*>(St);  // [2][64][kGradPitch]: dC, dB
    auto rows_sync = [] { asm volatile("bar.sync 1, 512;" ::: "memory"); };
    rows_sync();
    const int zr = 32 * (warp & 1) + lane, zc = 32 * (warp >> 2);  // row and 32 columns of Z1, Y1 (warps 0, 1 of four) or Z2, Y2
    for (int pass = 0; pass < 2; ++pass) {
      if (ok && ((warp >> 1) & 1) == 1 - pass) {
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          float f[32];
          ld_acc32(taddr + (which ? tY : tZ), warp, zc, f);
          float4* dst = reinterpret_cast<float4*>(Sum + (which * Q + zr) * kGradPitch + zc);
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            if (pass == 0) {  // J of the sine part
              dst[x] = make_float4(-f[4 * x + 1], f[4 * x], -f[4 * x + 3], f[4 * x + 2]);
            } else {
              const float4 o = dst[x];
              dst[x] = make_float4(o.x + f[4 * x], o.y + f[4 * x + 1], o.z + f[4 * x + 2], o.w + f[4 * x + 3]);
            }
          }
        }
      }
      rows_sync();
    }
    wait(m1, nh);
    tc::fence_after_sync();
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      const int c16 = 64 * ((warp >> 1) & 1) + 16 * (warp >> 2);
      const size_t ui = ((size_t)b * p.G * p.splits + blockIdx.y) * p.n + c;
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        float f[16];
        ld_acc16(taddr + (which ? tV : tU), warp, 16 * (warp >> 2), f);
        const float4* src = reinterpret_cast<const float4*>(Sum + (which * Q + t) * kGradPitch + c16);
        uint4* dst = reinterpret_cast<uint4*>((which ? p.pb : p.pc) + ui * (N * Q)) + t;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float4 o = src[x];
          f[4 * x] += o.x; f[4 * x + 1] += o.y; f[4 * x + 2] += o.z; f[4 * x + 3] += o.w;
        }
        dst[(c16 >> 3) * Q] = pack8(f);
        dst[((c16 >> 3) + 1) * Q] = pack8(f + 8);
      }
    }
    tc::fence_before_sync();
  }
  if (!ok && lane == 0) atomicExch(p.status, 13);
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 512);
}


// ------------------------------------------------------------ final per-token scalars
constexpr int kTailThreads = 512;
constexpr int kTailHeads = 32;   // heads of a scalar block

// ddt, dlambda, dtheta of the steps of a chunk and up to 32 heads, and their share of da_log.  The workspace has the steps of
// a head in a row, the caller's tensors the heads of a step: the latter go through shared memory, so that both sides move whole
// lines (a block per (batch, head) that walked the sequence read and wrote 4 bytes of every 32: 38 us at 8 x 4096 x 32 heads).
__device__ __forceinline__ void final_scalars(const SsdP& p, int block) {
  __shared__ float th[Q][kTailHeads + 1], dr[Q][kTailHeads + 1], dl[Q][kTailHeads + 1];  // theta -> dtheta, dt_raw -> ddt, dlambda
  __shared__ float wsum[2 * kTailHeads];
  const int groups = (p.NH + kTailHeads - 1) / kTailHeads, hg = block % groups, c = (block / groups) % p.n, b = block / groups / p.n;
  const int h0 = hg * kTailHeads, nh = min(kTailHeads, p.NH - h0), t0 = c * Q, nt = min(Q, p.T - t0);
  const int tid = threadIdx.x;
  const size_t row0 = ((size_t)b * p.T + t0) * p.NH + h0;
  for (int u = tid; u < Q * kTailHeads; u += kTailThreads) {
    const int t = u / kTailHeads, h = u % kTailHeads;
    const bool in = t < nt && h < nh;
    th[t][h] = in ? __ldg(p.theta + row0 + (size_t)t * p.NH + h) : 0.f;
    dr[t][h] = in ? __ldg(p.dt_raw + row0 + (size_t)t * p.NH + h) : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int u = tid; u < Q * kTailHeads; u += kTailThreads) {
    const int h = u / Q, t = u % Q;
    float dal = 0.f;
    if (t < nt && h < nh) {
      const size_t o = ((size_t)b * p.NH + h0 + h) * p.T + t0 + t;
      const float A = -expf(p.a_log[h0 + h]);
      const float dt = p.dt[o], lam = p.lam[o], da = p.da[o], dinc = p.dphi[o];
      const float dgam = p.dgam[o] + p.de[o], dnxt = t0 + t > 0 ? p.de[o - 1] : 0.f;
      const float ddelta = A * da + lam * dgam + (1.f - lam) * dnxt + th[t][h] * dinc;
      dr[t][h] = ddelta * sigmoid_f(dr[t][h]);
      dl[t][h] = dt * (dgam - dnxt) * lam * (1.f - lam);
      th[t][h] = dt * dinc;
      dal = A * dt * da;
    }
    dal = warp_sum(dal);  // (a warp has 32 steps of one head)
    if ((tid & 31) == 0) wsum[u >> 5] = dal;
  }
  __syncthreads();
  for (int u = tid; u < Q * kTailHeads; u += kTailThreads) {
    const int t = u / kTailHeads, h = u % kTailHeads;
    if (t < nt && h < nh) {
      const size_t r = row0 + (size_t)t * p.NH + h;
      p.ddt[r] = dr[t][h];
      p.dlam[r] = dl[t][h];
      p.dtheta[r] = th[t][h];
    }
  }
  if (tid < nh) p.dal_part[((size_t)b * p.n + c) * p.NH + h0 + tid] = wsum[2 * tid] + wsum[2 * tid + 1];
}
// dB[b,t,g,:] = sum over the partial images of group g (fp32, fixed order).  A thread owns eight
// states of a row; consecutive threads hold consecutive rows, which are neighbours in the column-blocked images.
__device__ __forceinline__ void reduce_rows(const bf16* __restrict__ pb, const bf16* __restrict__ pc, bf16* __restrict__ db,
                                            bf16* __restrict__ dc, int T, int G, int per, int n, int block) {
  static_assert(2 * kTailThreads == N / 8 * Q, "a block covers half of the states of a chunk and one gradient");
  const int which = (block >> 1) & 1, r = threadIdx.x & 63, c8 = (threadIdx.x >> 6) + 8 * (block & 1);
  int rest = block >> 2;
  const int c = rest % n;
  rest /= n;
  const int g = rest % G, b = rest / G, t = c * Q + r;
  if (t >= T) return;
  const uint4* src = reinterpret_cast<const uint4*>(which ? pc : pb) +
                     (((size_t)b * G + g) * per * n + c) * (N / 8 * Q) + c8 * Q + r;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int h = 0; h < per; ++h) {
    float e[8];
    unpack8(__ldg(src + (size_t)h * n * (N / 8 * Q)), e);
#pragma unroll
    for (int y = 0; y < 8; ++y) acc[y] += e[y];
  }
  *reinterpret_cast<uint4*>((which ? dc : db) + (((size_t)b * T + t) * G + g) * N + 8 * c8) = pack8(acc);
}

// The first nf blocks do the per-token scalars, the others the row sums: both read what the chunk kernel left.
__global__ void __launch_bounds__(kTailThreads, 3) m3s_tail_kernel(SsdP p, bf16* __restrict__ db, bf16* __restrict__ dc, int nf) {
  begin_dependent();
  const int block = blockIdx.x;
  if (block < nf) final_scalars(p, block);
  else reduce_rows(p.pb, p.pc, db, dc, p.T, p.G, p.splits, p.n, block - nf);
}
// A warp per head; the lanes' shares and their sum in a fixed order.
__global__ void __launch_bounds__(128) m3s_dalog_kernel(SsdP p) {
  begin_dependent();
  const int head = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (head >= p.NH) return;
  float s = 0.f;
#pragma unroll 4
  for (int u = lane; u < p.B * p.n; u += 32) s += p.dal_part[(size_t)u * p.NH + head];
  s = warp_sum(s);
  if (lane == 0) p.da_log[head] = s;
}

}  // namespace m3s

// ------------------------------------------------------------------ host
using m3s::SsdP;

bool mamba3_ssd_supported(const mxb_mamba3_desc* d) {
  if (d->io_dtype != MXB_BF16 || d->nheads <= 0 || d->D % d->nheads) return false;
  if (d->D / d->nheads != m3s::P || d->N != m3s::N) return false;
  if ((d->D / d->G) % m3s::P || d->nheads % d->G) return false;
  return true;
}

static size_t carve_ssd(SsdP& p, void* ws, bool bwd) {
  Carver cv(ws);
  const size_t bh = (size_t)p.B * p.NH, nst = bh * p.n * m3s::N * m3s::P;
  p.status = cv.take<int>(64);
  p.dt = cv.take<float>(bh * p.T);
  p.lam = cv.take<float>(bh * p.T);
  p.theta_t = cv.take<float>(bh * p.T);
  p.cs = cv.take<float>(bh * p.n * (sizeof(m3s::ChunkScal) / 4));
  p.H0 = cv.take<m3s::bf16>(nst);
  if (bwd) {
    p.dH1 = cv.take<m3s::bf16>(nst);
    p.dphi = cv.take<float>(bh * p.T);
    p.da = cv.take<float>(bh * p.T);
    p.de = cv.take<float>(bh * p.T);
    p.dgam = cv.take<float>(bh * p.T);
    p.dal_part = cv.take<float>(bh * p.n);
    const size_t images = (size_t)p.B * p.G * p.splits * p.n * m3s::Q * m3s::N;
    p.pb = cv.take<m3s::bf16>(images);
    p.pc = cv.take<m3s::bf16>(images);
  }
  return cv.bytes();
}

static SsdP make_ssd(const mxb_mamba3_desc* d) {
  SsdP p{};
  p.B = d->B; p.T = d->T; p.D = d->D; p.G = d->G; p.NH = d->nheads;
  p.n = (d->T + m3s::Q - 1) / m3s::Q;
  const int per = p.NH / p.G;
  // Heads per CTA of the chunk-gradient kernel: a CTA costs 7 us and 2.7 us a head, one runs per SM.  Not by the batch, so
  // that a sequence gives the same bits alone (the partial sums are rounded).  us with 16 / 8 / 4 / 2 heads, chunks x heads of
  // a sequence: 2048 (8 sequences) 361 / 406 / 676 / -; 512 (8) 105 / 117 / 129 / 174, (2) 54 / 34 / 41 / 54;
  // 256 (8) 56 / 64 / 76 / 93, (1) 53 / 33 / 23 / 17; 32 (1) - / 32 / 22 / 17.
  const int u = p.n * p.NH;
  p.hp = std::min(per, u >= 1024 ? 16 : u >= 512 ? 8 : u >= 256 ? 4 : 2);
  p.splits = (per + p.hp - 1) / p.hp;
  p.no_tma = (d->flags & MXB_MAMBA3_NO_TMA) ? 1 : 0;
  return p;
}

size_t mamba3_ssd_workspace_bytes(const mxb_mamba3_desc* d, bool bwd) {
  SsdP p = make_ssd(d);
  return carve_ssd(p, nullptr, bwd);
}

bool make_tma_map_bthd(CUtensorMap* m, const void* base, int B, int T, int H, int D);

// Tensor maps for the token-indexed operands of the chunk kernels (dy only in the backward); false when one
// cannot be made (no tensor-map entry point in the driver): the kernels then stage with cp.async.  Either way
// the operand bases are 16-byte aligned: the dispatcher refuses other pointers.
static bool ssd_chunk_maps(const SsdP& p, m3s::ChunkMaps& maps) {
  std::memset(&maps, 0, sizeof maps);
  if (p.no_tma) return false;
  bool ok = make_tma_map_bthd(&maps.b, p.b, p.B, p.T, p.G, m3s::N) && make_tma_map_bthd(&maps.c, p.c, p.B, p.T, p.G, m3s::N) &&
            make_tma_map_bthd(&maps.x, p.x, p.B, p.T, p.NH, m3s::P);
  if (ok && p.dy)
    ok = make_tma_map_bthd(&maps.dy, p.dy, p.B, p.T, p.NH, m3s::P) && make_tma_map_bthd(&maps.dx, p.dx, p.B, p.T, p.NH, m3s::P);
  return ok;
}

// Sequential pass over the chunks (mode 0: forward states, mode 1: reverse state gradients); the copy engine
// feeds it when tensor maps can be made for the operands, cp.async otherwise.
static mxb_status ssd_state_pass(SsdP& p, int mode, cudaStream_t st) {
  m3s::PassMaps maps;
  std::memset(&maps, 0, sizeof maps);
  const bool tma = !p.no_tma && make_tma_map_bthd(&maps.r, mode == 0 ? p.b : p.c, p.B, p.T, p.G, m3s::N) &&
                   make_tma_map_bthd(&maps.x, mode == 0 ? p.x : p.dy, p.B, p.T, p.NH, m3s::P);
  auto launch = [&](auto tma_v, auto ns) {
    constexpr bool TMA = decltype(tma_v)::value;
    constexpr int NS = decltype(ns)::value;
    if (MXB_ALLOW_SMEM(m3s::kPassSmem<NS>, m3s::m3s_state_pass_kernel<TMA, NS>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("m3s_state_pass_kernel", st,
               (launch_kernel(m3s::m3s_state_pass_kernel<TMA, NS>, dim3(p.NH, p.B), m3s::kPassThreads<NS>, m3s::kPassSmem<NS>, st, p, mode, maps)));
    return MXB_OK;
  };
  const std::integral_constant<int, 3> three;
  const std::integral_constant<int, 6> six;
  const bool alone = p.NH * p.B <= 148;  // every CTA has an SM of its own
  const mxb_status s = tma ? (alone ? launch(std::true_type{}, six) : launch(std::true_type{}, three))
                           : (alone ? launch(std::false_type{}, six) : launch(std::false_type{}, three));
  if (s != MXB_OK) return s;
  return check_launch("m3s_state_pass_kernel");
}

// States and output by one kernel where the CTAs of the state pass would share SMs; false where a tensor map cannot be made.  Of
// fewer (batch, head) pairs the chain of chunks is what counts, and the output kernel spreads over all SMs.  A forward with its
// scalars, us, two kernels / one that keeps the states / one that does not: 1 x 4096 x 32 heads 74 / 136 / 125, 4 x 4096 x 32 145 / 163
// / 158, 4 x 1024 x 37 47.7 / 51.2 / 51.3, 149 x 512 x 1 36.3 / 33.6 / 32.5, 5 x 512 x 30 34.6 / 32.3 / 31.5, 5 x 4096 x 32 213 / 220 /
// 204 (long sequences that keep their states lose a little at 160 pairs and gain at 192), 6 x 4096 x 32 237 / 225 / 209, 8 x 4096 x 32 284 / 235 / 213;
// in a second round of CTAs 9 x 4096 x 33 368 / 355 / 324, 10 x 2048 x 32 196 / 185 / 187, 16 x 2048 x 32 285 / 233 / 211.  The bits
// are the same.
static bool ssd_scan_maps(const SsdP& p, m3s::ScanMaps& maps) {
  std::memset(&maps, 0, sizeof maps);
  return !p.no_tma && make_tma_map_bthd(&maps.b, p.b, p.B, p.T, p.G, m3s::N) && make_tma_map_bthd(&maps.c, p.c, p.B, p.T, p.G, m3s::N) &&
         make_tma_map_bthd(&maps.x, p.x, p.B, p.T, p.NH, m3s::P) && make_tma_map_bthd(&maps.y, p.y, p.B, p.T, p.NH, m3s::P);
}

// save: the states at the chunk starts are kept for a backward.
static mxb_status ssd_forward(SsdP& p, bool save, cudaStream_t st) {
  const dim3 gc(p.n, p.NH, p.B);
  // (the chunks' shares of the angle lie where the state pass writes the chunk states afterwards)
  double* share = reinterpret_cast<double*>(p.H0);
  MXB_LAUNCH("m3s_scalars_kernel", st,
             (launch_kernel(m3s::m3s_scalars_kernel, dim3(p.n * ((p.NH + m3s::kScalHeads - 1) / m3s::kScalHeads), p.B), m3s::kScalThreads, 0, st, p, share)));
  const double* angles = share;
  // A block of the next kernel adds the shares of all chunks in front of its own: fine for short sequences, but it grows with the
  // square of their number.  Sums by a launch of their own from chunks^2 x heads of 2 M on (not by the batch: a sequence gives the
  // same bits alone).  Forward, us, without / with it, chunks x heads: 64 x 32 84 / 86, 128 x 32 161 / 162, 256 x 8 228 / 231,
  // 256 x 32 309 / 306 (4 sequences 599 / 587), 512 x 8 450 / 452, 1024 x 8 890 / 886, 512 x 32 607 / 596, 2048 x 32 2594 / 2364.
  if ((long long)p.n * p.n * p.NH >= 1 << 21) {
    MXB_LAUNCH("m3s_angle_prefix_kernel", st,
               (launch_kernel(m3s::m3s_angle_prefix_kernel, dim3((p.NH + m3s::kScalHeads - 1) / m3s::kScalHeads, p.B),
                              m3s::kScalHeads * m3s::kPrefixSegs, 0, st, p, share)));
    MXB_LAUNCH("m3s_chunk_scalars_kernel", st, (launch_kernel(m3s::m3s_chunk_scalars_kernel<true>, gc, 64, 0, st, p, angles)));
  } else {
    MXB_LAUNCH("m3s_chunk_scalars_kernel", st, (launch_kernel(m3s::m3s_chunk_scalars_kernel<false>, gc, 64, 0, st, p, angles)));
  }
  m3s::ScanMaps scan;
  if (p.y && p.NH * p.B > 148 && ssd_scan_maps(p, scan)) {
    if (MXB_ALLOW_SMEM(m3s::kScanSmem, m3s::m3s_scan_out_kernel) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("m3s_scan_out_kernel", st,
               (launch_kernel(m3s::m3s_scan_out_kernel, dim3(p.NH, p.B), m3s::kScanThreads, m3s::kScanSmem, st, p, save ? 1 : 0, scan)));
    return check_launch("mamba3 ssd forward");
  }
  mxb_status ps = ssd_state_pass(p, 0, st);
  if (ps != MXB_OK) return ps;
  if (p.y) {
    m3s::ChunkMaps maps;
    if (ssd_chunk_maps(p, maps)) {
      if (MXB_ALLOW_SMEM(m3s::kOutSmem, m3s::m3s_chunk_out_kernel<true>) != MXB_OK) return MXB_ERR_CUDA;
      MXB_LAUNCH("m3s_chunk_out_kernel", st, (launch_kernel(m3s::m3s_chunk_out_kernel<true>, gc, 128, m3s::kOutSmem, st, p, maps)));
    } else {
      if (MXB_ALLOW_SMEM(m3s::kOutSmem, m3s::m3s_chunk_out_kernel<false>) != MXB_OK) return MXB_ERR_CUDA;
      MXB_LAUNCH("m3s_chunk_out_kernel", st, (launch_kernel(m3s::m3s_chunk_out_kernel<false>, gc, 128, m3s::kOutSmem, st, p, maps)));
    }
  }
  return check_launch("mamba3 ssd forward");
}

mxb_status mamba3_ssd_fwd(const mxb_mamba3_desc* d, const void* x, const float* dt, const float* lam,
                          const float* theta, const float* a_log, const void* b, const void* c, void* y, void* ws,
                          cudaStream_t st) {
  SsdP p = make_ssd(d);
  p.x = static_cast<const m3s::bf16*>(x); p.b = static_cast<const m3s::bf16*>(b); p.c = static_cast<const m3s::bf16*>(c);
  p.dt_raw = dt; p.lam_raw = lam; p.theta = theta; p.a_log = a_log; p.y = static_cast<m3s::bf16*>(y);
  carve_ssd(p, ws, false);
  return ssd_forward(p, (d->flags & MXB_MAMBA3_SAVE_FOR_BWD) != 0, st);
}

mxb_status mamba3_ssd_bwd(const mxb_mamba3_desc* d, const void* x, const float* dt, const float* lam,
                          const float* theta, const float* a_log, const void* b, const void* c, const void* dy,
                          void* dx, float* ddt, float* dlam, float* dtheta, float* da_log, void* db, void* dc, void* ws,
                          cudaStream_t st) {
  SsdP p = make_ssd(d);
  p.x = static_cast<const m3s::bf16*>(x); p.b = static_cast<const m3s::bf16*>(b); p.c = static_cast<const m3s::bf16*>(c);
  p.dy = static_cast<const m3s::bf16*>(dy); p.dx = static_cast<m3s::bf16*>(dx);
  p.dt_raw = dt; p.lam_raw = lam; p.theta = theta; p.a_log = a_log;
  p.ddt = ddt; p.dlam = dlam; p.dtheta = dtheta; p.da_log = da_log;
  carve_ssd(p, ws, true);
  p.y = nullptr;  // the forward recompute stops at the chunk states
  // with saved intermediates dt, lambda, phi, the chunk decays and H0 are still in place
  if (!(d->flags & MXB_MAMBA3_BWD_USE_SAVED)) {
    mxb_status s = ssd_forward(p, true, st);
    if (s != MXB_OK) return s;
  }
  const dim3 gg(p.n, p.G * p.splits, p.B);
  mxb_status ps = ssd_state_pass(p, 1, st);
  if (ps != MXB_OK) return ps;
  m3s::ChunkMaps maps;
  if (ssd_chunk_maps(p, maps)) {
    if (MXB_ALLOW_SMEM(m3s::kGradSmem, m3s::m3s_chunk_grad_kernel<true>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("m3s_chunk_grad_kernel", st, (launch_kernel(m3s::m3s_chunk_grad_kernel<true>, gg, m3s::kGradThreads, m3s::kGradSmem, st, p, maps)));
  } else {
    if (MXB_ALLOW_SMEM(m3s::kGradSmem, m3s::m3s_chunk_grad_kernel<false>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("m3s_chunk_grad_kernel", st, (launch_kernel(m3s::m3s_chunk_grad_kernel<false>, gg, m3s::kGradThreads, m3s::kGradSmem, st, p, maps)));
  }
  const int nf = p.B * p.n * ((p.NH + m3s::kTailHeads - 1) / m3s::kTailHeads), tail = nf + 4 * p.n * p.G * p.B;
  MXB_LAUNCH("m3s_tail_kernel", st,
             (launch_kernel(m3s::m3s_tail_kernel, tail, m3s::kTailThreads, 0, st, p, static_cast<m3s::bf16*>(db), static_cast<m3s::bf16*>(dc), nf)));
  MXB_LAUNCH("m3s_dalog_kernel", st, (launch_kernel(m3s::m3s_dalog_kernel, (p.NH + 3) / 4, 128, 0, st, p)));
  return check_launch("mamba3 ssd backward");
}

}  // namespace mxb
