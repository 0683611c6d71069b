// Element-wise stages of mixlab's gated_deltanet block around the scan
// (emitGatedDeltaNetDeltaIR, arch/blocks_gated_deltanet.go:207-343; short convolution :345-368):
//   pre   q_seq = SiLU(conv4(q_proj)), k_seq = SiLU(conv4(k_proj)), v = SiLU(conv4(v_proj))      causal, 4 taps
//         q = q_seq rsqrt(mean(q_seq^2) + 1e-6) / dk,  k = k_seq rsqrt(mean(k_seq^2) + 1e-6) / sqrt(dk)
//         gate = exp(-softplus(a_raw + dt_bias) exp(A_log)),  beta = sigmoid(b_raw)
//   post  y = o rsqrt(mean(o^2) + 1e-5) o_norm SiLU(z)
// and their backward passes.  All of it is an HBM stream: every element is read once (plus a 3-step halo of the
// convolution) and written once, in 16-byte pieces.
//
// Work split: a row is one (batch, step, head) vector of D <= 128 channels; as many lanes as it needs (a power of two)
// cover it with 4 channels each (convolution stages) or 8 (output stage).
// Sums over (batch, step) - convolution weight, norm weight, A_log, dt_bias gradients - go through per-CTA partial
// rows in the workspace and a fixed-order second pass (no atomics).
#include <type_traits>

#include "common.cuh"
#include "packed.cuh"

namespace mxb {
namespace blk {

using bf16 = __nv_bfloat16;

struct BlockP {
  int B, T, H, Dk, Dv, gate_is_log;
};

template <typename IO>
__device__ __forceinline__ void load8(const IO* p, float (&e)[8]);
template <>
__device__ __forceinline__ void load8<float>(const float* p, float (&e)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w; e[4] = b.x; e[5] = b.y; e[6] = b.z; e[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<bf16>(const bf16* p, float (&e)[8]) {
  const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) { e[2 * i] = __low2float(h[i]); e[2 * i + 1] = __high2float(h[i]); }
}
template <typename IO>
__device__ __forceinline__ void store8(IO* p, const float (&e)[8]);
template <>
__device__ __forceinline__ void store8<float>(float* p, const float (&e)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(e[0], e[1], e[2], e[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(e[4], e[5], e[6], e[7]);
}
template <>
__device__ __forceinline__ void store8<bf16>(bf16* p, const float (&e)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(e[2 * i], e[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = v;
}
__device__ __forceinline__ float sigmoid_f(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }
// sigmoid for the streams: bf16 I/O takes tanh.approx (one MUFU op, relative error ~5e-4, far below the rounding
// of the stored result); fp32 I/O takes exp + reciprocal (a few ulp)
template <typename IO>
__device__ __forceinline__ float sigmoid_io(float x) {
  return sigmoid_f(x);
}
template <>
__device__ __forceinline__ float sigmoid_io<__nv_bfloat16>(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return fmaf(0.5f, t, 0.5f);
}
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

// which of the three streams (q, k, v) a CTA works on
template <typename IO>
struct PreArgs {
  const IO* x[3];        // q_proj, k_proj, v_proj   [B,T,H*D]
  const float* w[3];     // conv weights             [4, H*D]
  IO* y[3];              // q, k, v
  const IO* dy[3];       // backward: dq, dk, dv
  IO* dx[3];             // backward: dq_proj, dk_proj, dv_proj
  float* dwp[3];         // backward: per-CTA partial rows [B*ntiles][4][H*D]
};

// Four channels of a step as they come from memory, and widened to two packed pairs.
template <typename IO>
struct Raw4 { uint2 v; };
template <>
struct Raw4<float> { float4 v; };
__device__ __forceinline__ void load_raw(Raw4<bf16>& r, const bf16* p, bool ok) {
  r.v = ok ? __ldg(reinterpret_cast<const uint2*>(p)) : make_uint2(0u, 0u);
}
__device__ __forceinline__ void load_raw(Raw4<float>& r, const float* p, bool ok) {
  r.v = ok ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void widen(f2 (&e)[2], const Raw4<bf16>& r) {
  e[0] = pack2(__uint_as_float(r.v.x << 16), __uint_as_float(r.v.x & 0xffff0000u));
  e[1] = pack2(__uint_as_float(r.v.y << 16), __uint_as_float(r.v.y & 0xffff0000u));
}
__device__ __forceinline__ void widen(f2 (&e)[2], const Raw4<float>& r) {
  e[0] = pack2(r.v.x, r.v.y);
  e[1] = pack2(r.v.z, r.v.w);
}
__device__ __forceinline__ void store_pairs(bf16* p, const f2 (&e)[2]) {
  const float2 a = unpack2(e[0]), b = unpack2(e[1]);
  __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(b.x, b.y);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
__device__ __forceinline__ void store_pairs(float* p, const f2 (&e)[2]) {
  const float2 a = unpack2(e[0]), b = unpack2(e[1]);
  *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
}
template <typename IO>
__device__ __forceinline__ f2 sigmoid_pair(f2 x) {
  const float2 a = unpack2(x);
  return pack2(sigmoid_io<IO>(a.x), sigmoid_io<IO>(a.y));
}
template <>
__device__ __forceinline__ f2 sigmoid_pair<bf16>(f2 x) {
  float2 a = unpack2(mul2(x, dup2(0.5f)));
  asm("tanh.approx.f32 %0, %0;" : "+f"(a.x));
  asm("tanh.approx.f32 %0, %0;" : "+f"(a.y));
  return mad2(pack2(a.x, a.y), dup2(0.5f), dup2(0.5f));
}
// Backward: ring of steps (x and dy) in shared memory between the copies (cp.async) and the arithmetic, every thread on
// its own four channels: no barriers, and three batches of four steps in flight without holding registers (244 -> 205 us
// for 16 x 2048 x 16 heads of 64 bf16 channels; the forward, which has registers to spare, is faster without: 84, 89 us).
template <typename IO>
struct PreRing {
  static constexpr int kStages = sizeof(IO) == 2 ? 4 : 2;  // (two CTAs per SM)
  static constexpr int kUnit = 4 * sizeof(IO), kBatch = 4 * 2 * 256 * kUnit, kBytes = kStages * kBatch;
  uint32_t base;
  __device__ __forceinline__ explicit PreRing(const void* smem)
      : base(static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + threadIdx.x * kUnit) {}
  __device__ __forceinline__ uint32_t at(int batch, int tensor, int s) const {
    return base + (batch & (kStages - 1)) * kBatch + (tensor * 4 + s) * 256 * kUnit;
  }
  // size: kUnit, or 0 for zeros (src must be a mapped address all the same)
  __device__ __forceinline__ void copy(uint32_t dst, const IO* src, uint32_t size) const {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(kUnit), "r"(size) : "memory");
  }
  static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  static __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory"); }
  __device__ __forceinline__ void get(int batch, int tensor, int s, f2 (&e)[2]) const {
    Raw4<IO> r;
    if constexpr (sizeof(IO) == 2)
      asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.v.x), "=r"(r.v.y) : "r"(at(batch, tensor, s)) : "memory");
    else
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.v.x), "=f"(r.v.y), "=f"(r.v.z), "=f"(r.v.w)
                   : "r"(at(batch, tensor, s)) : "memory");
    widen(e, r);
  }
};
// Row sums of four steps at once over the LPR lanes of a row: lane l ends up with the sum of step l & 3.  Halving
// exchanges: 3 + log2(LPR / 4) shuffles instead of 4 log2(LPR).
template <int LPR>
__device__ __forceinline__ float row_sums4(const float (&v)[4]) {
  const int l = threadIdx.x;
  const bool b0 = l & 1, b1 = l & 2;
  const float u0 = (b0 ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[1], 1);
  const float u1 = (b0 ? v[3] : v[2]) + __shfl_xor_sync(0xffffffffu, b0 ? v[2] : v[3], 1);
  float s = (b1 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b1 ? u0 : u1, 2);
#pragma unroll
  for (int o = 4; o < LPR; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
// A value that lane l holds for step l & 3, for step s.
__device__ __forceinline__ float of_step(float v, int s) { return __shfl_sync(0xffffffffu, v, (threadIdx.x & 28) | s); }

// Thread map of the convolution stages: a CTA of 256 threads covers 64 x 4 channels of consecutive heads (LPR lanes per
// row of a head; one contiguous piece of a time step) and four runs of `run` consecutive steps.  Steps go in batches
// of four, the loads of the next batch (backward: of the next three) in flight behind the arithmetic of the current one;
// the previous three inputs (and, backward, the previous three ds) stay in registers.
constexpr int kPreRuns = 4;
struct PreMap {
  int head, ch, t0;
  bool act;
  template <int LPR>
  static __device__ __forceinline__ PreMap make(int H, int D, int run) {
    const int seg = threadIdx.x & 63, l = seg & (LPR - 1);
    PreMap m;
    m.head = blockIdx.x * (64 / LPR) + seg / LPR;
    m.act = m.head < H && 4 * l < D;
    m.ch = m.head * D + 4 * l;
    m.t0 = (blockIdx.y * kPreRuns + (threadIdx.x >> 6)) * run;
    return m;
  }
};

// ------------------------------------------------------------------ pre: forward
// grid (head blocks, time tiles, streams x B from z0 on)
template <typename IO, int LPR>
__global__ void __launch_bounds__(256) gdn_block_pre_fwd_kernel(BlockP p, PreArgs<IO> a, int run, int first, int z0) {
  begin_dependent();
  const int which = first + (z0 + blockIdx.z) / p.B, b = (z0 + blockIdx.z) % p.B;
  const int D = which == 2 ? p.Dv : p.Dk, C = p.H * D;
  const PreMap m = PreMap::make<LPR>(p.H, D, run);
  const IO* x = a.x[which] + (size_t)b * p.T * C + m.ch;
  IO* y = a.y[which] + (size_t)b * p.T * C + m.ch;
  f2 w[4][2];  // zero for the lanes beyond D: their zero results take part in the row sums
#pragma unroll
  for (int tap = 0; tap < 4; ++tap) {
    Raw4<float> r;
    load_raw(r, a.w[which] + tap * C + m.ch, m.act);
    widen(w[tap], r);
  }
  const float inv_d = 1.f / (float)D, scale = which == 0 ? inv_d : rsqrtf((float)D);  // q: 1/dk, k: 1/sqrt(dk)
  auto fetch = [&](Raw4<IO>& r, int t) { load_raw(r, x + (size_t)t * C, m.act && t >= 0 && t < p.T); };
  f2 xx[7][2];  // inputs of the steps t-3 .. t+3
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Raw4<IO> r;
    fetch(r, m.t0 - 3 + k);
    widen(xx[k], r);
  }
  Raw4<IO> nx[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) fetch(nx[s], m.t0 + s);
  for (int r0 = 0; r0 < run; r0 += 4) {
    const int t = m.t0 + r0;
#pragma unroll
    for (int s = 0; s < 4; ++s) widen(xx[3 + s], nx[s]);
    if (r0 + 4 < run) {
#pragma unroll
      for (int s = 0; s < 4; ++s) fetch(nx[s], t + 4 + s);
    }
    f2 sv[4][2];
    float ss[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      f2 sq = 0ull;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        f2 acc = mul2(w[0][c], xx[s + 3][c]);
        fma2(acc, w[1][c], xx[s + 2][c]);
        fma2(acc, w[2][c], xx[s + 1][c]);
        fma2(acc, w[3][c], xx[s][c]);
        sv[s][c] = mul2(acc, sigmoid_pair<IO>(acc));
        fma2(sq, sv[s][c], sv[s][c]);
      }
      ss[s] = sum2(sq);
    }
    if (which < 2) {
      const float rn = rsqrtf(fmaf(row_sums4<LPR>(ss), inv_d, 1e-6f)) * scale;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const f2 f = dup2(of_step(rn, s));
        sv[s][0] = mul2(sv[s][0], f);
        sv[s][1] = mul2(sv[s][1], f);
      }
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (m.act && t + s < p.T) store_pairs(y + (size_t)(t + s) * C, sv[s]);
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) xx[j][c] = xx[j + 4][c];
  }
}

// gate = exp(-softplus(a_raw + dt_bias) exp(A_log)) (or its log), beta = sigmoid(b_raw): one thread per (b, t, h)
__global__ void __launch_bounds__(256) gdn_block_gate_fwd_kernel(BlockP p, const float* __restrict__ a_raw,
                                                                 const float* __restrict__ b_raw,
                                                                 const float* __restrict__ a_log,
                                                                 const float* __restrict__ dt_bias,
                                                                 float* __restrict__ beta, float* __restrict__ gate) {
  begin_dependent();
  const size_t n = (size_t)p.B * p.T * p.H;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
    const int h = (int)(i % p.H);
    const float lg = -softplus_f(a_raw[i] + dt_bias[h]) * expf(a_log[h]);
    gate[i] = p.gate_is_log ? lg : expf(lg);
    beta[i] = sigmoid_f(b_raw[i]);
  }
}

// ------------------------------------------------------------------ pre: backward
// Same map as the forward.  A run recomputes the convolution of its steps and of the three steps after it (their ds
// feeds dx of the run) and emits dx three steps behind.  Bound: HBM (nine tensors) and, close behind, issue: about
// 17 instructions per element with packed arithmetic (40 and half of the lanes idle at 64 channels before: 760 us for
// 16 x 2048 x 16 heads of 64 bf16 channels, 182 now).  Two CTAs per SM leave a thread 128 registers for its weights, weight
// gradients, seven inputs and seven ds of four channels, so little else may live across the row sums: two products with the
// derivative of SiLU instead of SiLU, derivative and dy (180 bytes spilled: 198 us; 24 now).
template <typename IO, int LPR>
__global__ void __launch_bounds__(256, 2) gdn_block_pre_bwd_kernel(BlockP p, PreArgs<IO> a, int run, int first, int z0) {
  begin_dependent();
  extern __shared__ __align__(16) uint8_t pre_smem[];
  __shared__ float red[kPreRuns][4][256];
  const int which = first + (z0 + blockIdx.z) / p.B, b = (z0 + blockIdx.z) % p.B;
  const int D = which == 2 ? p.Dv : p.Dk, C = p.H * D;
  const PreMap m = PreMap::make<LPR>(p.H, D, run);
  const IO* x = a.x[which] + (size_t)b * p.T * C + m.ch;
  const IO* dy = a.dy[which] + (size_t)b * p.T * C + m.ch;
  IO* dx = a.dx[which] + (size_t)b * p.T * C + m.ch;
  f2 w[4][2], dw[4][2];
#pragma unroll
  for (int tap = 0; tap < 4; ++tap) {
    Raw4<float> r;
    load_raw(r, a.w[which] + tap * C + m.ch, m.act);
    widen(w[tap], r);
    dw[tap][0] = dw[tap][1] = 0ull;
  }
  const float inv_d = 1.f / (float)D, scale = which == 0 ? inv_d : rsqrtf((float)D);
  auto fetch = [&](Raw4<IO>& r, const IO* src, int t) { load_raw(r, src + (size_t)t * C, m.act && t >= 0 && t < p.T); };
  f2 xx[7][2], dd[7][2];  // inputs and ds of the steps t-3 .. t+3
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Raw4<IO> r;
    fetch(r, x, m.t0 - 3 + k);
    widen(xx[k], r);
    dd[k][0] = dd[k][1] = 0ull;
  }
  const PreRing<IO> ring(pre_smem);
  const int batches = run / 4;
  // Copies of batch k: pointers advance by four steps; a step past the end re-reads the last one with size zero, and so
  // do lanes without channels.
  const IO *cx = m.act ? x : a.x[which], *cg = m.act ? dy : a.dy[which];
  const uint32_t size = m.act ? ring.kUnit : 0;
  const size_t stride = m.act ? C : 0;
  const bool full = m.t0 + run + 4 <= p.T;  // every copy and every result of this run lies inside the sequence
  cx += (size_t)min(m.t0, p.T - 1) * stride;
  cg += (size_t)min(m.t0, p.T - 1) * stride;
  auto issue = [&](int k) {
    if (k <= batches) {
      const uint32_t d0 = ring.at(k, 0, 0), d1 = ring.at(k, 1, 0);
      if (full) {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          ring.copy(d0 + s * 256 * ring.kUnit, cx + s * stride, size);
          ring.copy(d1 + s * 256 * ring.kUnit, cg + s * stride, size);
        }
        cx += 4 * stride;
        cg += 4 * stride;
      } else {
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int t = m.t0 + 4 * k + s;
          ring.copy(d0 + s * 256 * ring.kUnit, cx, t < p.T ? size : 0);
          ring.copy(d1 + s * 256 * ring.kUnit, cg, t < p.T ? size : 0);
          if (t + 1 < p.T) {
            cx += stride;
            cg += stride;
          }
        }
      }
    }
    ring.commit();
  };
  IO* ox = dx + (size_t)m.t0 * C - (size_t)3 * C;  // dx of step t0 + 4 k - 3
#pragma unroll
  for (int k = 0; k < ring.kStages - 1; ++k) issue(k);
  for (int k = 0; k <= batches; ++k) {  // the last batch is the halo: three steps, no weight gradient
    const int r0 = 4 * k;
    const bool halo = k == batches;
    f2 g[4][2];
    ring.wait();
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      ring.get(k, 0, s, xx[3 + s]);
      ring.get(k, 1, s, g[s]);
    }
    issue(k + ring.kStages - 1);
    // one sigmoid per element gives SiLU and its derivative; rows past T have zero dy, hence zero ds
    f2 sv[4][2];  // SiLU times its derivative (g: the same of dy): what a row sum away becomes ds
    float ss[4], dot[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      f2 sq = 0ull, sg_dot = 0ull;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        f2 acc = mul2(w[0][c], xx[s + 3][c]);
        fma2(acc, w[1][c], xx[s + 2][c]);
        fma2(acc, w[2][c], xx[s + 1][c]);
        fma2(acc, w[3][c], xx[s][c]);
        const f2 sg = sigmoid_pair<IO>(acc);
        const f2 si = mul2(acc, sg), dsl = mad2(si, mad2(sg, dup2(-1.f), dup2(1.f)), sg);  // dsl = sg (1 + acc (1 - sg))
        fma2(sq, si, si);
        fma2(sg_dot, si, g[s][c]);
        sv[s][c] = mul2(si, dsl);
        g[s][c] = mul2(g[s][c], dsl);
      }
      ss[s] = sum2(sq);
      dot[s] = sum2(sg_dot);
    }
    if (which < 2) {  // y = s rn scale: gradient at s = scale rn (g - s rn^2 dot / D)
      const float rn = rsqrtf(fmaf(row_sums4<LPR>(ss), inv_d, 1e-6f));
      const float fa = scale * rn, fb = -fa * rn * rn * (row_sums4<LPR>(dot) * inv_d);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const f2 f0 = dup2(of_step(fa, s)), f1 = dup2(of_step(fb, s));
#pragma unroll
        for (int c = 0; c < 2; ++c) dd[3 + s][c] = mad2(f1, sv[s][c], mul2(f0, g[s][c]));
      }
    } else {
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int c = 0; c < 2; ++c) dd[3 + s][c] = g[s][c];
    }
    if (!halo) {
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int tap = 0; tap < 4; ++tap)
#pragma unroll
          for (int c = 0; c < 2; ++c) fma2(dw[tap][c], xx[s + 3 - tap][c], dd[3 + s][c]);
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {  // dx of step t+s-3: w0 ds[t+s-3] + ... + w3 ds[t+s]
      const int r = r0 + s - 3;
      if (m.act && (s == 3 ? !halo : k > 0) && (full || m.t0 + r < p.T)) {
        f2 o[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          o[c] = mul2(w[0][c], dd[s][c]);
          fma2(o[c], w[1][c], dd[s + 1][c]);
          fma2(o[c], w[2][c], dd[s + 2][c]);
          fma2(o[c], w[3][c], dd[s + 3][c]);
        }
        store_pairs(ox + (size_t)s * C, o);
      }
    }
    ox += (size_t)4 * C;
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        xx[j][c] = xx[j + 4][c];
        dd[j][c] = dd[j + 4][c];
      }
  }
  // weight-gradient partial of this CTA: its four runs added in a fixed order
  const int seg = threadIdx.x & 63, rid = threadIdx.x >> 6;
#pragma unroll
  for (int tap = 0; tap < 4; ++tap) {
    const float2 lo = unpack2(dw[tap][0]), hi = unpack2(dw[tap][1]);
    *reinterpret_cast<float4*>(&red[rid][tap][4 * seg]) = make_float4(lo.x, lo.y, hi.x, hi.y);
  }
  __syncthreads();
  if (m.act) {  // thread = tap rid, its own four channels
    float4 s = *reinterpret_cast<const float4*>(&red[0][rid][4 * seg]);
#pragma unroll
    for (int k = 1; k < kPreRuns; ++k) {
      const float4 v = *reinterpret_cast<const float4*>(&red[k][rid][4 * seg]);
      s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
    }
    *reinterpret_cast<float4*>(a.dwp[which] + (((size_t)b * gridDim.y + blockIdx.y) * 4 + rid) * C + m.ch) = s;
  }
}

// out[j] = sum over rows of part[row][j] in a fixed order.  Up to five matrices per launch, segment s starting at block first[s].
struct ColSums {
  const float* part[5];
  float* out[5];
  int rows[5], n[5], first[6], count;
};
template <bool TALL>
__global__ void __launch_bounds__(kSumThreads<TALL>) gdn_block_colsum_kernel(ColSums c) {
  begin_dependent();
  int g = 0;
  while (g + 1 < c.count && (int)blockIdx.x >= c.first[g + 1]) ++g;
  const int n = c.n[g], j0 = (blockIdx.x - c.first[g]) * kSumCols<TALL>, mine = j0 + threadIdx.x % kSumCols<TALL>;
  float* out = c.out[g];
  col_sum<TALL>(c.part[g] + mine, c.rows[g], n, mine < n, [&](int x, float t) {
    if (j0 + x < n) out[j0 + x] = t;
  });
}

// gate / beta backward: one CTA per head walks all (b, t); the two per-head sums (A_log, dt_bias) in a fixed order
__global__ void __launch_bounds__(256) gdn_block_gate_bwd_kernel(BlockP p, const float* __restrict__ a_raw,
                                                                 const float* __restrict__ b_raw,
                                                                 const float* __restrict__ a_log,
                                                                 const float* __restrict__ dt_bias,
                                                                 const float* __restrict__ dbeta,
                                                                 const float* __restrict__ dgate,
                                                                 float* __restrict__ da_raw, float* __restrict__ db_raw,
                                                                 float* __restrict__ da_log, float* __restrict__ ddt_bias) {
  begin_dependent();
  __shared__ float red[2][8];
  const int h = blockIdx.x, tid = threadIdx.x;
  const float A = expf(a_log[h]), bias = dt_bias[h];
  float s_alog = 0.f, s_bias = 0.f;
  const int n = p.B * p.T;
  for (int i = tid; i < n; i += 256) {
    const size_t idx = (size_t)i * p.H + h;
    const float z = a_raw[idx] + bias;
    const float lg = -softplus_f(z) * A;
    const float dlg = p.gate_is_log ? dgate[idx] : dgate[idx] * expf(lg);
    const float da = -A * dlg * sigmoid_f(z);
    da_raw[idx] = da;
    s_bias += da;
    s_alog = fmaf(dlg, lg, s_alog);  // d lg / d A_log = lg
    const float bt = sigmoid_f(b_raw[idx]);
    db_raw[idx] = dbeta[idx] * bt * (1.f - bt);
  }
  s_alog = warp_sum(s_alog);
  s_bias = warp_sum(s_bias);
  if ((tid & 31) == 0) { red[0][tid >> 5] = s_alog; red[1][tid >> 5] = s_bias; }
  __syncthreads();
  if (tid == 0) {
    float x = 0.f, y = 0.f;
    for (int w = 0; w < 8; ++w) { x += red[0][w]; y += red[1][w]; }
    da_log[h] = x;
    ddt_bias[h] = y;
  }
}

// The same with every (b, t, h) element on its own thread, coalesced, for head counts that divide 256: a thread's
// head is then tid % H for every element it touches.  Per-CTA partial sums [2][G][H] -> fixed-order second pass.
constexpr int kGatePerCta = 256 * 8;
__global__ void __launch_bounds__(256) gdn_block_gate_bwd_flat_kernel(BlockP p, const float* __restrict__ a_raw,
                                                                      const float* __restrict__ b_raw,
                                                                      const float* __restrict__ a_log,
                                                                      const float* __restrict__ dt_bias,
                                                                      const float* __restrict__ dbeta,
                                                                      const float* __restrict__ dgate,
                                                                      float* __restrict__ da_raw,
                                                                      float* __restrict__ db_raw,
                                                                      float* __restrict__ part) {
  begin_dependent();
  __shared__ float red[2][256];
  const int tid = threadIdx.x, h = tid % p.H;
  const float A = expf(a_log[h]), bias = dt_bias[h];
  const size_t n = (size_t)p.B * p.T * p.H, base = (size_t)blockIdx.x * kGatePerCta;
  const size_t end = base + kGatePerCta < n ? base + kGatePerCta : n;
  float s_alog = 0.f, s_bias = 0.f;
  for (size_t idx = base + tid; idx < end; idx += 256) {
    const float z = a_raw[idx] + bias;
    const float lg = -softplus_f(z) * A;
    const float dlg = p.gate_is_log ? dgate[idx] : dgate[idx] * expf(lg);
    const float da = -A * dlg * sigmoid_f(z);
    da_raw[idx] = da;
    s_bias += da;
    s_alog = fmaf(dlg, lg, s_alog);
    const float bt = sigmoid_f(b_raw[idx]);
    db_raw[idx] = dbeta[idx] * bt * (1.f - bt);
  }
  red[0][tid] = s_alog;
  red[1][tid] = s_bias;
  __syncthreads();
  if (tid < p.H) {
    float x = 0.f, y = 0.f;
    for (int j = tid; j < 256; j += p.H) { x += red[0][j]; y += red[1][j]; }
    part[(size_t)blockIdx.x * p.H + tid] = x;
    part[((size_t)gridDim.x + blockIdx.x) * p.H + tid] = y;
  }
}

// ------------------------------------------------------------------ post
// y = o rsqrt(mean(o^2) + 1e-5) o_norm SiLU(z); rows = (b, t, h), D = Dv.  A thread owns 8 channels, LPR lanes a row
// (with 16 lanes for every width, half of them idled at 64 channels: 60 us instead of 36 for 16 x 2048 x 16 rows);
// two rows per pass, so that the loads of both are in flight.
template <int LPR>
__device__ __forceinline__ float lane_sum(float v) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename IO, int LPR>
__global__ void __launch_bounds__(128) gdn_block_post_fwd_kernel(BlockP p, const IO* __restrict__ o,
                                                                 const IO* __restrict__ z,
                                                                 const float* __restrict__ wn, IO* __restrict__ y) {
  begin_dependent();
  constexpr int kRows = 128 / LPR;  // rows of a CTA
  const int D = p.Dv, l = threadIdx.x % LPR;
  const bool act = l * 8 < D;
  const size_t rows = (size_t)p.B * p.T * p.H, step = (size_t)gridDim.x * kRows;
  float w[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (act) load8<float>(wn + l * 8, w);
  for (size_t first = (size_t)blockIdx.x * kRows; first < rows; first += 2 * step) {
    float ov[2][8], zv[2][8];
    bool in[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const size_t row = first + u * step + threadIdx.x / LPR;
      in[u] = act && row < rows;
#pragma unroll
      for (int c = 0; c < 8; ++c) ov[u][c] = zv[u][c] = 0.f;
      if (in[u]) { load8<IO>(o + row * D + l * 8, ov[u]); load8<IO>(z + row * D + l * 8, zv[u]); }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const size_t row = first + u * step + threadIdx.x / LPR;
      float ss = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) ss = fmaf(ov[u][c], ov[u][c], ss);
      const float rn = rsqrtf(lane_sum<LPR>(ss) / (float)D + 1e-5f);
#pragma unroll
      for (int c = 0; c < 8; ++c) ov[u][c] = ov[u][c] * rn * w[c] * zv[u][c] * sigmoid_io<IO>(zv[u][c]);
      if (in[u]) store8<IO>(y + row * D + l * 8, ov[u]);
    }
  }
}

template <typename IO, int LPR>
__global__ void __launch_bounds__(128) gdn_block_post_bwd_kernel(BlockP p, const IO* __restrict__ o,
                                                                 const IO* __restrict__ z,
                                                                 const float* __restrict__ wn,
                                                                 const IO* __restrict__ dy, IO* __restrict__ d_o,
                                                                 IO* __restrict__ dz, float* __restrict__ dwp) {
  begin_dependent();
  constexpr int kRows = 128 / LPR;
  __shared__ float red[kRows][8 * LPR];
  const int D = p.Dv, l = threadIdx.x % LPR;
  const bool act = l * 8 < D;
  const size_t rows = (size_t)p.B * p.T * p.H, step = (size_t)gridDim.x * kRows;
  float w[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, dw[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (act) load8<float>(wn + l * 8, w);
  for (size_t first = (size_t)blockIdx.x * kRows; first < rows; first += step) {
    const size_t row = first + threadIdx.x / LPR, off = row * D + l * 8;
    const bool in = act && row < rows;
    float ov[8], zv[8], gv[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) ov[c] = zv[c] = gv[c] = 0.f;
    if (in) { load8<IO>(o + off, ov); load8<IO>(z + off, zv); load8<IO>(dy + off, gv); }
    float ss = 0.f, dot = 0.f, g[8], sz[8], dsz[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float sg = sigmoid_io<IO>(zv[c]);
      sz[c] = zv[c] * sg;
      dsz[c] = fmaf(sz[c], 1.f - sg, sg);
      g[c] = gv[c] * sz[c] * w[c];  // gradient at o rn
      ss = fmaf(ov[c], ov[c], ss);
      dot = fmaf(ov[c], g[c], dot);
    }
    const float rn = rsqrtf(lane_sum<LPR>(ss) / (float)D + 1e-5f);
    const float k2 = rn * rn * lane_sum<LPR>(dot) / (float)D;
    float dzv[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float on = ov[c] * rn;
      dw[c] = fmaf(gv[c] * sz[c], on, dw[c]);
      dzv[c] = gv[c] * w[c] * on * dsz[c];
      g[c] = rn * (g[c] - ov[c] * k2);
    }
    if (in) { store8<IO>(d_o + off, g); store8<IO>(dz + off, dzv); }
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) red[threadIdx.x / LPR][l * 8 + c] = dw[c];
  __syncthreads();
  for (int c = threadIdx.x; c < D; c += 128) {
    float s = 0.f;
#pragma unroll
    for (int g2 = 0; g2 < kRows; ++g2) s += red[g2][c];
    dwp[(size_t)blockIdx.x * D + c] = s;
  }
}

}  // namespace blk

// ------------------------------------------------------------------ host
using blk::BlockP;

static BlockP make_blk(const mxb_gdn_desc* d) {
  BlockP p{};
  p.B = d->B; p.T = d->T; p.H = d->H; p.Dk = d->Dk; p.Dv = d->Dv; p.gate_is_log = d->gate_is_log;
  return p;
}
bool gdn_block_supported(const mxb_gdn_desc* d) {
  return d->Dk % 8 == 0 && d->Dv % 8 == 0 && d->Dk <= 128 && d->Dv <= 128 && d->Dk > 0 && d->Dv > 0;
}
// Lanes per row: the power of two that covers D / per channels.
static int blk_lanes(int D, int per) {
  int l = per == 4 ? 4 : 1;
  while (l * per < D) l *= 2;
  return l;
}
// Steps per run: 32 (a halo of three steps is recomputed per run in the backward) while that still gives two CTAs per
// SM, shorter runs for smaller problems, where the length of the chain is what counts.  Longer ones where the tiles of a
// sequence would not fit a grid axis.
static int blk_run(const mxb_gdn_desc* d) {
  const int hk = 64 / blk_lanes(d->Dk, 4);
  int longest = 32;
  while (d->T / (4 * longest) >= 65535) longest *= 2;
  if (longest > 32) return longest;
  for (int run = 32; run > 4; run /= 2)
    if ((size_t)3 * d->B * ((d->H + hk - 1) / hk) * ((d->T + 4 * run - 1) / (4 * run)) >= 2 * 148) return run;
  return 4;
}
static int blk_tiles(const mxb_gdn_desc* d) {
  const int tile = blk::kPreRuns * blk_run(d);
  return (d->T + tile - 1) / tile;
}
// CTAs of the output stage: what is on the GPU at once (eight an SM forward, six backward: 61 to 64 and 76 to 78 registers in every
// variant, 128 threads), so that no second round of a few CTAs follows (backward, 16 x 2048 x 16 heads of 64: 73 us with eight an SM
// asked for, 60 with six).
static int blk_post_ctas(const mxb_gdn_desc* d, bool bwd) {
  const size_t rows = (size_t)d->B * d->T * d->H, per = 128 / blk_lanes(d->Dv, 8);
  const size_t want = (rows + per - 1) / per, most = 148 * (bwd ? 6 : 8);
  return (int)(want < most ? want : most);
}
static int blk_gate_ctas(const mxb_gdn_desc* d) {
  const size_t n = (size_t)d->B * d->T * d->H;
  return (int)((n + blk::kGatePerCta - 1) / blk::kGatePerCta);
}
// backward partial rows: conv weights of q, k, v and the per-head gate sums; or the norm weight
size_t gdn_block_workspace_bytes(const mxb_gdn_desc* d) {
  const size_t rows = (size_t)d->B * blk_tiles(d);
  const size_t pre = rows * 4 * ((size_t)2 * d->H * d->Dk + (size_t)d->H * d->Dv) * sizeof(float);
  const size_t post = (size_t)blk_post_ctas(d, true) * d->Dv * sizeof(float);
  const size_t gate = 2 * (size_t)blk_gate_ctas(d) * d->H * sizeof(float);
  return (pre + gate > post ? pre + gate : post) + 256;
}

// call(LPR) with the lane count as a compile-time constant
template <typename F>
static void with_lanes(int lanes, F&& call) {
  switch (lanes) {
    case 1: call(std::integral_constant<int, 1>{}); break;
    case 2: call(std::integral_constant<int, 2>{}); break;
    case 4: call(std::integral_constant<int, 4>{}); break;
    case 8: call(std::integral_constant<int, 8>{}); break;
    case 16: call(std::integral_constant<int, 16>{}); break;
    default: call(std::integral_constant<int, 32>{}); break;
  }
}
// The convolution kernels over q, k (streams 0, 1) and v (2): one launch where the lane counts agree, two otherwise, and
// more where the sequences of all streams do not fit a grid axis.
constexpr int kGridZ = 65535;
template <typename F>
static void blk_streams(const mxb_gdn_desc* d, F&& launch) {
  const int lk = blk_lanes(d->Dk, 4), lv = blk_lanes(d->Dv, 4), nt = blk_tiles(d);
  auto over = [&](int lanes, int streams, int first) {
    for (int z0 = 0; z0 < streams * d->B; z0 += kGridZ) {
      const int nz = streams * d->B - z0 < kGridZ ? streams * d->B - z0 : kGridZ;
      launch(lanes, dim3((d->H + 64 / lanes - 1) / (64 / lanes), nt, nz), first, z0);
    }
  };
  over(lk, lk == lv ? 3 : 2, 0);
  if (lk != lv) over(lv, 1, 2);
}

template <typename IO>
static mxb_status blk_pre_fwd(const mxb_gdn_desc* d, const void* qp, const void* kp, const void* vp, const float* cq,
                              const float* ck, const float* cv, const float* a_raw, const float* b_raw,
                              const float* a_log, const float* dt_bias, void* q, void* k, void* v, float* beta,
                              float* gate, cudaStream_t st) {
  BlockP p = make_blk(d);
  blk::PreArgs<IO> a{};
  a.x[0] = static_cast<const IO*>(qp); a.x[1] = static_cast<const IO*>(kp); a.x[2] = static_cast<const IO*>(vp);
  a.w[0] = cq; a.w[1] = ck; a.w[2] = cv;
  a.y[0] = static_cast<IO*>(q); a.y[1] = static_cast<IO*>(k); a.y[2] = static_cast<IO*>(v);
  const int run = blk_run(d);
  blk_streams(d, [&](int lanes, dim3 grid, int first, int z0) {
    with_lanes(lanes, [&](auto lpr) {
      constexpr int LPR = decltype(lpr)::value;
      if constexpr (LPR >= 4)
        MXB_LAUNCH("gdn_block_pre_fwd_kernel", st, (launch_kernel(blk::gdn_block_pre_fwd_kernel<IO, LPR>, grid, 256, 0, st, p, a, run, first, z0)));
    });
  });
  const size_t n = (size_t)d->B * d->T * d->H;
  const int gb = (int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
  MXB_LAUNCH("gdn_block_gate_fwd_kernel", st,
             (launch_kernel(blk::gdn_block_gate_fwd_kernel, gb, 256, 0, st, p, a_raw, b_raw, a_log, dt_bias, beta, gate)));
  return check_launch("gdn_block_pre_fwd");
}
mxb_status gdn_block_pre_fwd(const mxb_gdn_desc* d, const void* qp, const void* kp, const void* vp, const float* cq,
                             const float* ck, const float* cv, const float* a_raw, const float* b_raw,
                             const float* a_log, const float* dt_bias, void* q, void* k, void* v, float* beta,
                             float* gate, cudaStream_t st) {
  return d->io_dtype == MXB_F32
             ? blk_pre_fwd<float>(d, qp, kp, vp, cq, ck, cv, a_raw, b_raw, a_log, dt_bias, q, k, v, beta, gate, st)
             : blk_pre_fwd<blk::bf16>(d, qp, kp, vp, cq, ck, cv, a_raw, b_raw, a_log, dt_bias, q, k, v, beta, gate, st);
}

static void blk_colsum(blk::ColSums& c, cudaStream_t st) {
  size_t columns = 0;
  for (int i = 0; i < c.count; ++i) columns += c.n[i];
  auto launch = [&](auto tall) {
    constexpr bool TALL = decltype(tall)::value;
    for (int i = 0; i < c.count; ++i) c.first[i + 1] = c.first[i] + (c.n[i] + kSumCols<TALL> - 1) / kSumCols<TALL>;
    MXB_LAUNCH("gdn_block_colsum_kernel", st,
               (launch_kernel(blk::gdn_block_colsum_kernel<TALL>, c.first[c.count], kSumThreads<TALL>, 0, st, c)));
  };
  if (col_sum_tall(columns)) launch(std::true_type{});
  else launch(std::false_type{});
}

template <typename IO>
static mxb_status blk_pre_bwd(const mxb_gdn_desc* d, const void* qp, const void* kp, const void* vp, const float* cq,
                              const float* ck, const float* cv, const float* a_raw, const float* b_raw,
                              const float* a_log, const float* dt_bias, const void* dq, const void* dk, const void* dv,
                              const float* dbeta, const float* dgate, void* dqp, void* dkp, void* dvp, float* dcq,
                              float* dck, float* dcv, float* da_raw, float* db_raw, float* da_log, float* ddt_bias,
                              void* ws, cudaStream_t st) {
  BlockP p = make_blk(d);
  blk::PreArgs<IO> a{};
  a.x[0] = static_cast<const IO*>(qp); a.x[1] = static_cast<const IO*>(kp); a.x[2] = static_cast<const IO*>(vp);
  a.w[0] = cq; a.w[1] = ck; a.w[2] = cv;
  a.dy[0] = static_cast<const IO*>(dq); a.dy[1] = static_cast<const IO*>(dk); a.dy[2] = static_cast<const IO*>(dv);
  a.dx[0] = static_cast<IO*>(dqp); a.dx[1] = static_cast<IO*>(dkp); a.dx[2] = static_cast<IO*>(dvp);
  const int run = blk_run(d);
  const size_t rows = (size_t)d->B * blk_tiles(d), Ck = (size_t)d->H * d->Dk, Cv = (size_t)d->H * d->Dv;
  float* base = reinterpret_cast<float*>(static_cast<char*>(ws) + 256);
  a.dwp[0] = base; a.dwp[1] = base + rows * 4 * Ck; a.dwp[2] = base + rows * 8 * Ck;
  mxb_status s = MXB_OK;
  blk_streams(d, [&](int lanes, dim3 grid, int first, int z0) {
    with_lanes(lanes, [&](auto lpr) {
      constexpr int LPR = decltype(lpr)::value;
      if constexpr (LPR >= 4) {
        if (s == MXB_OK) s = MXB_ALLOW_SMEM(blk::PreRing<IO>::kBytes, blk::gdn_block_pre_bwd_kernel<IO, LPR>);
        if (s == MXB_OK)
          MXB_LAUNCH("gdn_block_pre_bwd_kernel", st,
                     (launch_kernel(blk::gdn_block_pre_bwd_kernel<IO, LPR>, grid, 256, blk::PreRing<IO>::kBytes, st, p, a, run, first, z0)));
      }
    });
  });
  if (s != MXB_OK) return s;
  blk::ColSums c{};
  auto sum = [&](const float* part, int nrows, int n, float* out) {
    c.part[c.count] = part; c.out[c.count] = out; c.rows[c.count] = nrows; c.n[c.count] = n;
    ++c.count;
  };
  sum(a.dwp[0], (int)rows, (int)(4 * Ck), dcq);
  sum(a.dwp[1], (int)rows, (int)(4 * Ck), dck);
  sum(a.dwp[2], (int)rows, (int)(4 * Cv), dcv);
  if (256 % d->H == 0) {
    const int gc = blk_gate_ctas(d);
    float* gpart = base + rows * 4 * (2 * Ck + Cv);
    MXB_LAUNCH("gdn_block_gate_bwd_flat_kernel", st,
               (launch_kernel(blk::gdn_block_gate_bwd_flat_kernel, gc, 256, 0, st, p, a_raw, b_raw, a_log, dt_bias, dbeta, dgate,
                                                                       da_raw, db_raw, gpart)));
    sum(gpart, gc, d->H, da_log);
    sum(gpart + (size_t)gc * d->H, gc, d->H, ddt_bias);
  } else {
    MXB_LAUNCH("gdn_block_gate_bwd_kernel", st,
               (launch_kernel(blk::gdn_block_gate_bwd_kernel, d->H, 256, 0, st, p, a_raw, b_raw, a_log, dt_bias, dbeta, dgate,
                                                                      da_raw, db_raw, da_log, ddt_bias)));
  }
  blk_colsum(c, st);
  return check_launch("gdn_block_pre_bwd");
}
mxb_status gdn_block_pre_bwd(const mxb_gdn_desc* d, const void* qp, const void* kp, const void* vp, const float* cq,
                             const float* ck, const float* cv, const float* a_raw, const float* b_raw,
                             const float* a_log, const float* dt_bias, const void* dq, const void* dk, const void* dv,
                             const float* dbeta, const float* dgate, void* dqp, void* dkp, void* dvp, float* dcq,
                             float* dck, float* dcv, float* da_raw, float* db_raw, float* da_log, float* ddt_bias,
                             void* ws, cudaStream_t st) {
  return d->io_dtype == MXB_F32
             ? blk_pre_bwd<float>(d, qp, kp, vp, cq, ck, cv, a_raw, b_raw, a_log, dt_bias, dq, dk, dv, dbeta, dgate, dqp,
                                  dkp, dvp, dcq, dck, dcv, da_raw, db_raw, da_log, ddt_bias, ws, st)
             : blk_pre_bwd<blk::bf16>(d, qp, kp, vp, cq, ck, cv, a_raw, b_raw, a_log, dt_bias, dq, dk, dv, dbeta, dgate,
                                      dqp, dkp, dvp, dcq, dck, dcv, da_raw, db_raw, da_log, ddt_bias, ws, st);
}

template <typename IO>
static mxb_status blk_post(const mxb_gdn_desc* d, const void* o, const void* z, const float* wn, void* y,
                           const void* dy, void* d_o, void* dz, float* dwn, void* ws, cudaStream_t st) {
  BlockP p = make_blk(d);
  const int ctas = blk_post_ctas(d, dy != nullptr);
  const int lanes = blk_lanes(d->Dv, 8);
  if (!dy) {
    with_lanes(lanes, [&](auto lpr) {
      constexpr int LPR = decltype(lpr)::value;
      if constexpr (LPR <= 16)
        MXB_LAUNCH("gdn_block_post_fwd_kernel", st,
                   (launch_kernel(blk::gdn_block_post_fwd_kernel<IO, LPR>, ctas, 128, 0, st, p, static_cast<const IO*>(o), static_cast<const IO*>(z), wn, static_cast<IO*>(y))));
    });
    return check_launch("gdn_block_post_fwd");
  }
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + 256);
  with_lanes(lanes, [&](auto lpr) {
    constexpr int LPR = decltype(lpr)::value;
    if constexpr (LPR <= 16)
      MXB_LAUNCH("gdn_block_post_bwd_kernel", st,
                 (launch_kernel(blk::gdn_block_post_bwd_kernel<IO, LPR>, ctas, 128, 0, st, p, static_cast<const IO*>(o), static_cast<const IO*>(z), wn, static_cast<const IO*>(dy),
                     static_cast<IO*>(d_o), static_cast<IO*>(dz), part)));
  });
  blk::ColSums c{};
  c.part[0] = part; c.out[0] = dwn; c.rows[0] = ctas; c.n[0] = d->Dv; c.count = 1;
  blk_colsum(c, st);
  return check_launch("gdn_block_post_bwd");
}
mxb_status gdn_block_post(const mxb_gdn_desc* d, const void* o, const void* z, const float* wn, void* y, const void* dy,
                          void* d_o, void* dz, float* dwn, void* ws, cudaStream_t st) {
  return d->io_dtype == MXB_F32 ? blk_post<float>(d, o, z, wn, y, dy, d_o, dz, dwn, ws, st)
                                : blk_post<blk::bf16>(d, o, z, wn, y, dy, d_o, dz, dwn, ws, st);
}

}  // namespace mxb
