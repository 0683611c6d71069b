// Mamba-3 selective scan, per-channel layout, window-parallel: forward and backward for problems whose (batch, channel)
// pairs cannot fill the GPU with walks over the whole sequence (mamba3.cu has the recurrence and the serial walk).
//
// A walker owns one (batch, channel, window of 8 steps).  Every carried quantity is linear in what crosses a window
// boundary, so the walk splits into local walks and scans over the windows:
//   prepare   softplus(dt), sigmoid(lambda) of every (step, channel), window sums of dt theta and dt
//   scan      angle at each window start
//   local     walks from a zero state (forward) and from a zero dh (reverse; backward only)
//   scan      H <- exp(A sum dt) H + local: state at each window start; the same for dh, in reverse (what enters a window is
//             also what the trapezoid's look-back sends to the window's last step: exp(A dt) up of the step behind)
//   walk      forward: the true walk writes y;  backward: replay into shared memory, then the true reverse walk with
//             window-local angle-gradient sums
//   sums, fix reverse scan of those sums (and the sums of dB, dC and da_log over CTAs and windows); the later windows' sums are
//             added to ddt and dtheta
//
// What bounds it: instruction issue (a sine, a cosine and two exponentials per state pair and pass).  So everything
// that belongs to a (step, channel) is computed once and not by every lane and pass; the two states of a pair and two
// pairs per lane go through packed arithmetic; a pass keeps sine and cosine (the local walk the decay too) in shared memory
// for its reverse half; rows of dB, dC are added over the channels of a warp by halving exchanges and over the warps once per
// window.  Scans run 32 segments of windows side by side.  2 x 1024 x 128 channels of 16 states, forward + backward:
// 71 us a call; 4096 x 448 channels: 140 us forward, 313 a backward with its recompute.
//
// Every sum has a fixed order: the same inputs give the same bits.
#include <algorithm>
#include <type_traits>

#include "mamba3.cuh"
#include "packed.cuh"

namespace mxb {
namespace m3w {

constexpr int W = kM3WinSteps;

// sin, cos of two angles in [-pi, pi] (a little more is fine): reduction by the nearest multiple of pi/2 in two parts
// (Cody and Waite), Taylor polynomials of degree 9 and 10 on [-pi/4, pi/4].  Truncation is below 2e-9.  Rounding: the
// reduced angle is off by at most 6e-8 (two roundings of a value below 0.79), which the sine takes over times its cosine
// and the cosine times its sine; the polynomials and their last addition add at most 5e-8: below 1.2e-7 together, as
// tests/test_mamba3_gpu.py checks over 16 million angles through mxb_selftest_sincos.
__device__ __forceinline__ void sincos2(f2 x, f2& sn, f2& cs) {
  const f2 magic = dup2(12582912.f), minus = dup2(-12582912.f);  // 1.5 * 2^23: rounds to the nearest integer
  const f2 kf = mad2(x, dup2(0.63661977236758134f), magic);
  const f2 k = add2(kf, minus);
  f2 r = mad2(k, dup2(-1.5707963705062866f), x);   // pi/2 rounded to float, and what is left of it
  r = mad2(k, dup2(4.3711390001862426e-8f), r);
  const f2 r2 = mul2(r, r);
  f2 ps = dup2(2.7557319223985893e-6f);
  ps = mad2(ps, r2, dup2(-1.9841269841269841e-4f));
  ps = mad2(ps, r2, dup2(8.3333333333333333e-3f));
  ps = mad2(ps, r2, dup2(-1.6666666666666667e-1f));
  ps = mad2(mul2(ps, r2), r, r);
  f2 pc = dup2(-2.7557319223985888e-7f);
  pc = mad2(pc, r2, dup2(2.4801587301587302e-5f));
  pc = mad2(pc, r2, dup2(-1.3888888888888889e-3f));
  pc = mad2(pc, r2, dup2(4.1666666666666667e-2f));
  pc = mad2(pc, r2, dup2(-0.5f));
  pc = mad2(pc, r2, dup2(1.f));
  const float2 s = unpack2(ps), c = unpack2(pc), q = unpack2(kf);
  auto quadrant = [](float s, float c, float q, float& so, float& co) {
    const int k = __float_as_int(q);  // the low bits of the rounded sum are the multiple of pi/2
    const float a = (k & 1) ? c : s, b = (k & 1) ? s : c;
    so = __int_as_float(__float_as_int(a) ^ ((k & 2) << 30));
    co = __int_as_float(__float_as_int(b) ^ (((k + 1) & 2) << 30));
  };
  float s0, c0, s1, c1;
  quadrant(s.x, c.x, q.x, s0, c0);
  quadrant(s.y, c.y, q.y, s1, c1);
  sn = pack2(s0, s1);
  cs = pack2(c0, c1);
}
// Two angles wrapped to [-pi, pi] (m3_wrap, packed).
__device__ __forceinline__ f2 wrap2(f2 x) {
  const f2 k = add2(mad2(x, dup2(0.15915494309189535f), dup2(12582912.f)), dup2(-12582912.f));
  return mad2(k, dup2(-1.9353071795864769e-3f), mad2(k, dup2(-6.28125f), x));
}
__global__ void __launch_bounds__(256) m3w_sincos_kernel(const float* __restrict__ x, size_t n, float* __restrict__ sn,
                                                         float* __restrict__ cs) {
  begin_dependent();
  for (size_t i = 2 * (blockIdx.x * (size_t)blockDim.x + threadIdx.x); i < n; i += 2 * (size_t)gridDim.x * blockDim.x) {
    const bool two = i + 1 < n;
    f2 s, c;
    sincos2(pack2(x[i], two ? x[i + 1] : 0.f), s, c);
    const float2 sv = unpack2(s), cv = unpack2(c);
    sn[i] = sv.x;
    cs[i] = cv.x;
    if (two) {
      sn[i + 1] = sv.y;
      cs[i + 1] = cv.y;
    }
  }
}
__device__ __forceinline__ f2 neg2(f2 v) { return v ^ 0x8000000080000000ull; }
// exp(dt a) of two states.  (One ex2 of a product with rates in base 2 would save 1 to 11 % of a call and is less exact: rms distance
// from float64 9.3e-8 for 6.8e-8 at exponents of 1 to 4, 3.5e-7 for 2.2e-7 at 4 to 16.)
__device__ __forceinline__ f2 decay2(f2 a, f2 dt) {
  const float2 x = unpack2(mul2(a, dt));
  return pack2(expf(x.x), expf(x.y));
}

// One walker: the lanes of one channel in one window.  A lane owns PR state pairs kp = sl PR + r in units of two; a
// packed value holds the same quantity of both pairs of a unit, even and odd states apart, so that the rotations are
// plain packed multiply-adds.  Whatever a window needs from global memory is requested before the first step: per-step
// scalars by the lane that owns the step (handed round by shuffles), theta into registers, the rows of b and c into
// shared memory, where all channels of the CTA read them.  Steps past the end of the sequence read as zeros, which
// leaves state and gradients untouched; only their results are not stored.
// PLAIN: per-channel parameters and rows that can be read two pairs at a time, known when compiled.
template <typename IO, int PR, int LPC, bool PLAIN>
struct Walker {
  static constexpr int CPW = 32 / LPC;             // channels per warp
  static constexpr int OWN = (W + LPC - 1) / LPC;  // steps whose scalars a lane holds
  static constexpr int UN = PR / 2;                // units of two pairs
  static constexpr int NP = PR * LPC;              // pairs per row, padded
  static constexpr int kRows = 2 * W + 1;          // rows in shared memory: b of ts-1 .. ts+W-1, then c of ts ..
  const M3P& p;
  const M3Idx ix;
  const bool vec, per_head;
  const int lane, sl, wc, d, b, w, ts, base;
  const size_t row0;
  float* rows;  // [kRows][2 (even, odd)][NP]
  __device__ Walker(const M3P& p_, float* rows_)
      : p(p_), ix(p_, PLAIN ? 0 : p_.NH), vec(PLAIN || p_.vec), per_head(!PLAIN && p_.NH > 0), lane(threadIdx.x & 31), sl(lane % LPC), wc((threadIdx.x >> 5) * CPW + lane / LPC),
        d(blockIdx.x * ((blockDim.x >> 5) * CPW) + wc), b(blockIdx.z), w(p_.w0 + blockIdx.y), ts(w * W), base(lane / LPC * LPC),
        row0((size_t)b * p_.T + ts), rows(rows_) {}
  __device__ bool act(int r) const { return sl * PR + r < p.Kp; }
  __device__ bool in(int s) const { return ts + s < p.T; }
  __device__ size_t wrow() const { return ((size_t)b * p.nW + w) * p.D + d; }
  __device__ size_t chan(int s) const { return ix.chan(row0 + s, d); }
  // per-step scalars: own(f)[o] = f(step sl + LPC o) for the steps inside the sequence; of(v, s): step s's value
  template <typename F>
  __device__ void own(float (&v)[OWN], F f) const {
#pragma unroll
    for (int o = 0; o < OWN; ++o) {
      const int s = sl + LPC * o;
      v[o] = s < W && in(s) ? f(s) : 0.f;
    }
  }
  __device__ float of(const float (&v)[OWN], int s) const { return __shfl_sync(0xffffffffu, v[s / LPC], base + s % LPC); }
  __device__ void stage(bool with_c) const {
    const IO *B = static_cast<const IO*>(p.b), *C = static_cast<const IO*>(p.c);
    const int n = with_c ? kRows : W + 1;
    const int d0 = blockIdx.x * ((blockDim.x >> 5) * CPW);  // any channel of the CTA: they share a group
    for (int u = threadIdx.x; u < n * NP; u += blockDim.x) {
      const int i = u / NP, kp = u - i * NP, t = i <= W ? ts - 1 + i : ts + i - W - 1;
      float e = 0.f, o = 0.f;
      if (kp < p.Kp && t >= 0 && t < p.T) {
        const IO* src = (i <= W ? B : C) + ix.grp((size_t)b * p.T + t, d0, 2 * kp);
        e = to_f32(src[0]);
        o = to_f32(src[1]);
      }
      rows[i * 2 * NP + kp] = e;
      rows[i * 2 * NP + NP + kp] = o;
    }
  }
  // row i of the staged rows in the frame of the angles: (c e + s o, c o - s e)
  __device__ void rotated(int i, int u, f2 sn, f2 cs, f2& v0, f2& v1) const {
    const f2 e = *reinterpret_cast<const f2*>(rows + i * 2 * NP + sl * PR + 2 * u);
    const f2 o = *reinterpret_cast<const f2*>(rows + i * 2 * NP + NP + sl * PR + 2 * u);
    v0 = mad2(sn, o, mul2(cs, e));
    v1 = mad2(neg2(sn), e, mul2(cs, o));
  }
  __device__ void rot_b(int s, int u, f2 sn, f2 cs, f2& v0, f2& v1) const { rotated(s + 1, u, sn, cs, v0, v1); }  // step ts + s
  __device__ void rot_c(int s, int u, f2 sn, f2 cs, f2& v0, f2& v1) const { rotated(W + 1 + s, u, sn, cs, v0, v1); }
  // one value per pair, from a row of Kp
  __device__ f2 two(const float* s, int u) const {
    s += sl * PR + 2 * u;
    if (vec) {
      if (!act(2 * u)) return 0ull;
      const float2 x = *reinterpret_cast<const float2*>(s);
      return pack2(x.x, x.y);
    }
    return pack2(act(2 * u) ? s[0] : 0.f, act(2 * u + 1) ? s[1] : 0.f);
  }
  __device__ void put_two(float* s, int u, f2 v) const {
    const float2 x = unpack2(v);
    s += sl * PR + 2 * u;
    if (vec) {
      if (act(2 * u)) *reinterpret_cast<float2*>(s) = x;
      return;
    }
    if (act(2 * u)) s[0] = x.x;
    if (act(2 * u + 1)) s[1] = x.y;
  }
  __device__ void thetas(f2 (&th)[W][UN]) const {
    const size_t stride = per_head ? p.NH : (size_t)p.D * p.Kp;
    const float* src = p.theta + ix.theta(row0, d, 0);
#pragma unroll
    for (int s = 0; s < W; ++s)
#pragma unroll
      for (int u = 0; u < UN; ++u) th[s][u] = !in(s) ? 0ull : per_head ? dup2(src[s * stride]) : two(src + s * stride, u);
  }
  // a row of N states: even (v0) and odd (v1) states of a unit
  __device__ void states(const float* s, int u, f2& v0, f2& v1) const {
    s += 2 * (sl * PR + 2 * u);
    if (vec) {
      const float4 x = act(2 * u) ? *reinterpret_cast<const float4*>(s) : make_float4(0.f, 0.f, 0.f, 0.f);
      v0 = pack2(x.x, x.z);
      v1 = pack2(x.y, x.w);
      return;
    }
    v0 = pack2(act(2 * u) ? s[0] : 0.f, act(2 * u + 1) ? s[2] : 0.f);
    v1 = pack2(act(2 * u) ? s[1] : 0.f, act(2 * u + 1) ? s[3] : 0.f);
  }
  __device__ void put_states(float* s, int u, f2 v0, f2 v1) const {
    const float2 x = unpack2(v0), y = unpack2(v1);
    s += 2 * (sl * PR + 2 * u);
    if (vec) {
      if (act(2 * u)) *reinterpret_cast<float4*>(s) = make_float4(x.x, y.x, x.y, y.y);
      return;
    }
    if (act(2 * u)) { s[0] = x.x; s[1] = y.x; }
    if (act(2 * u + 1)) { s[2] = x.y; s[3] = y.y; }
  }
  __device__ void rates(f2 (&A)[PR]) const {  // decay rates; A[2 u]: even states of unit u, A[2 u + 1]: odd
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      float a[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) a[x] = act(2 * u + x / 2) ? -expf(p.a_log[ix.alog(d, 2 * (sl * PR + 2 * u) + x)]) : 0.f;
      A[2 * u] = pack2(a[0], a[2]);
      A[2 * u + 1] = pack2(a[1], a[3]);
    }
  }
  // rotated b of the step before the window, at the window's start angle
  __device__ void before(const f2 (&phi)[UN], f2 (&pb)[PR]) const {
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      f2 sn, cs;
      sincos2(phi[u], sn, cs);
      rot_b(-1, u, sn, cs, pb[2 * u], pb[2 * u + 1]);
    }
  }
};
template <int PR, int LPC>
constexpr int kRowBytes = (2 * W + 1) * 2 * PR * LPC * 4;

// ------------------------------------------------------------------ prepare
// CTAs an SM: seven (32 registers) of four lanes a channel, or where rows are read two pairs at a time (4096 x 448 channels 2 us less
// than with 56 registers, 65 x 64 channels of 6 states 0.7); five (48 registers) of more lanes (18 to 128 states, against 32 registers
// and against no bound: up to 4 % of a forward); no bound with four pairs a lane, whose CTAs have at most
// 128 threads (256 states, 512 steps of 256 channels 248 us, 252 with 32 registers and 156 bytes spilled).
template <typename IO, int PR, int LPC, bool PLAIN>
__global__ void __launch_bounds__(256, LPC == 4 || PLAIN ? 7 : PR == 4 ? 1 : 5) m3w_prepare_kernel(M3P p) {
  begin_dependent();
  using K = Walker<IO, PR, LPC, PLAIN>;
  const K k(p, nullptr);
  f2 th[W][K::UN], ph[K::UN];
  k.thetas(th);
  const bool store = !k.per_head || k.d % k.ix.cph == 0;
  float dts[K::OWN];
  k.own(dts, [&](int s) {
    const size_t i = k.chan(s);
    const float v = m3_softplus(p.dt[i]);
    if (store) {
      p.dtv[i] = v;
      p.lamv[i] = m3_sigmoid(p.lam[i]);
    }
    return v;
  });
  float sum = 0.f;
#pragma unroll
  for (int u = 0; u < K::UN; ++u) ph[u] = 0ull;
#pragma unroll
  for (int s = 0; s < W; ++s) {
    const float dt = k.of(dts, s);
    sum += dt;
#pragma unroll
    for (int u = 0; u < K::UN; ++u) ph[u] = mad2(dup2(dt), th[s][u], ph[u]);
  }
#pragma unroll
  for (int u = 0; u < K::UN; ++u) k.put_two(p.ck_phi + k.wrow() * p.Kp, u, ph[u]);
  if (k.sl == 0) p.dtsum[k.wrow()] = sum;
}

// -------------------------------------------------------------------- scans
// 16 chains x 32 segments of PER windows per CTA: a segment is loaded once and folded, the folds of the earlier segments give
// what enters it, and the registers are walked again to write (longer sequences in rounds of 32 PER windows).  Latency and, with
// a decay, its exponentials bound it.  4096 x 448 channels of 16 states, us: one linear scan / both 20.5 / 51 with every value
// loaded twice and two or three exponentials, 19.5 / 33 without, 15.6 a scan since two CTAs of 64 registers share an SM.
//   kPhase  ck_phi: window sums -> wrapped angle at each window start, summed in 32-bit turns: additions that wrap by themselves and
//           do not round, of terms good to 1.5e-9.  The rounding of float sums, wrapped one by one, was a good part of the
//           distance of every result from float64 (900 steps: y 4.2e-7, dtheta 1.25e-6; 3.4e-7 and 9.8e-7 now)
//   kState  ck_h: local end states -> state at each window start
//   kDh     dhk: local dh -> dh entering each window from later steps
//   kAngle  ang: window sums -> sum over all later windows
enum { kPhase, kState, kDh, kAngle };
// An angle in units of 2^-32 of a turn: the rounded product, and what its rounding left, each to the nearest integer (1.5e-9 of
// angle together).  64 bits, of which the upper half are whole turns, hold window sums of up to 1.3e10, where a float no longer
// knows its angle; one wrapped to 32 bits in float before is rounded by up to 1e-7, or cut off where it comes out above pi.
__device__ __forceinline__ uint32_t turns(float x) {
  const float p = x * 683565248.f, e = fmaf(x, 27.5764316f, fmaf(x, 683565248.f, -p));
  return (uint32_t)__float2ll_rn(p) + (uint32_t)__float2ll_rn(e);
}
// The sum of angles: turns, and 0 or, once an angle was not finite, NaN: integers carry no NaN, and every later window has one.
struct Angle {
  uint32_t turns;
  float bad;
};
__device__ __forceinline__ Angle operator+(Angle a, Angle b) { return {a.turns + b.turns, a.bad + b.bad}; }
constexpr int kChains = 16, kSegs = 32, kScanThreads = kChains * kSegs;
template <int MODE, int PER>
__device__ __forceinline__ void scan_chain(const M3P& p, int chains, int block, int b) {
  constexpr bool linear = MODE == kState || MODE == kDh, back = MODE == kDh || MODE == kAngle;
  using Sum = std::conditional_t<MODE == kPhase, Angle, float>;
  __shared__ Sum s_add[kSegs][kChains];
  __shared__ float s_dec[kSegs][kChains];
  const int lane = threadIdx.x % kChains, seg = threadIdx.x / kChains, i = block * kChains + lane;
  const bool in = i < chains;
  float* buf = MODE == kPhase ? p.ck_phi : MODE == kState ? p.ck_h : MODE == kDh ? p.dhk : p.ang;
  const int d = linear ? i / p.N : 0;
  const float A = linear && in ? -expf(p.a_log[M3Idx(p).alog(d, i % p.N)]) : 0.f;
  auto win = [&](int x) { return (size_t)b * p.nW + (back ? p.nW - 1 - x : x); };  // x-th window in walking order
  auto value = [](float x) -> Sum {
    if constexpr (MODE == kPhase) return {turns(x), 0.f * x};
    else return x;
  };
  auto result = [](Sum run) -> float {
    if constexpr (MODE == kPhase) return fmaf((float)(int)run.turns, 1.4629180792671596e-9f, run.bad);  // 2 pi / 2^32
    else return run;
  };
  auto fold = [](float dec, Sum run, Sum add) -> Sum {
    if constexpr (linear) return fmaf(dec, run, add);
    else return run + add;
  };
  Sum carry{};
  for (int x0 = 0; x0 < p.nW; x0 += kSegs * PER) {
    const int lo = x0 + seg * PER;
    Sum loc[PER];
    float dec[PER];
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      const bool ok = in && lo + x < p.nW;
      loc[x] = value(ok ? buf[win(lo + x) * chains + i] : 0.f);
      dec[x] = ok && linear ? p.dtsum[win(lo + x) * p.D + d] : 0.f;
    }
    Sum run{};
    float dts = 0.f;
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      dts += dec[x];
      if (linear) dec[x] = expf(A * dec[x]);
      run = fold(dec[x], run, loc[x]);
    }
    s_add[seg][lane] = run;
    if (linear) s_dec[seg][lane] = expf(A * dts);
    __syncthreads();
    run = carry;
    const bool last = x0 + kSegs * PER >= p.nW;
    const int upto = last ? min(seg + 1, (p.nW - x0 + PER - 1) / PER) : kSegs;  // what comes behind enters no window
    for (int s0 = 0; s0 < upto; s0 += 8) {  // (eight reads ahead of the chain; all 32 segments cost short sequences 1 us a scan)
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        if (s0 + x == seg) carry = run;
        run = fold(linear ? s_dec[s0 + x][lane] : 0.f, run, s_add[s0 + x][lane]);
      }
    }
    const Sum through = run;
    run = carry;
    carry = through;
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      if (in && lo + x < p.nW) buf[win(lo + x) * chains + i] = result(run);
      run = fold(dec[x], run, loc[x]);
    }
    __syncthreads();
  }
}
template <int PER>
__global__ void __launch_bounds__(kScanThreads, 2) m3w_phase_scan_kernel(M3P p) {
  begin_dependent();
  scan_chain<kPhase, PER>(p, p.D * p.Kp, blockIdx.x, blockIdx.y);
}
// What follows the gradient walk and does not wait for each other, in one launch (three took 12 us at 2 x 1024 x 128 channels,
// 5 together): the first `scans` blocks scan the angle gradients, the next `dalogs` add the shares of da_log, the others
// the rows of dB and dC.
template <typename IO, int PER>
__global__ void __launch_bounds__(kScanThreads) m3w_sums_kernel(M3P p, int scans, int dalogs) {
  static_assert(kScanThreads == 32 * kDalogSlices, "one block size");
  begin_dependent();
  const int block = blockIdx.x;
  if (block < scans) scan_chain<kAngle, PER>(p, p.D * p.Kp, block / p.B, block % p.B);
  else if (block < scans + dalogs) m3_dalog_sum(p, p.B * p.nW, block - scans);
  else m3_bc_sum<IO>(p, block - scans - dalogs, gridDim.x - scans - dalogs);
}
// blockIdx.z: 0 the states, 1 dh (first: the one to start with)
template <int PER>
__global__ void __launch_bounds__(kScanThreads, 2) m3w_linear_scan_kernel(M3P p, int first) {
  begin_dependent();
  if (first + (int)blockIdx.z == 0) scan_chain<kState, PER>(p, p.D * p.N, blockIdx.x, blockIdx.y);
  else scan_chain<kDh, PER>(p, p.D * p.N, blockIdx.x, blockIdx.y);
}

// -------------------------------------------------------------- local walks
// Forward from a zero state (leaves the end state in ck_h) and, with DH, back with dh alone:
//   up_t = dh_t + dy_t Crot_t,  dh_{t-1} = alpha_t up_t
// (leaves the dh that leaves the window at its start in dhk).  Sine, cosine and decay of a step wait in shared memory for the
// way back.
template <typename IO, int PR, int LPC, bool PLAIN, bool FWD, bool DH>
__global__ void __launch_bounds__(256) m3w_local_kernel(M3P p) {
  begin_dependent();
  using K = Walker<IO, PR, LPC, PLAIN>;
  constexpr int UN = K::UN;
  extern __shared__ f2 hist[];  // [W][2 PR][threads], then the rows
  const K k(p, reinterpret_cast<float*>(hist + (DH ? W * 2 * PR * blockDim.x : 0)));
  auto slot = [&](int s, int x) -> f2& { return hist[(s * (2 * PR) + x) * blockDim.x + threadIdx.x]; };
  const IO *X = static_cast<const IO*>(p.x), *DY = static_cast<const IO*>(p.dy);
  f2 th[W][UN], phi[UN], A[PR];
  k.thetas(th);
  float dts[K::OWN], lams[K::OWN], xs[K::OWN], dys[K::OWN], px = 0.f;
  k.own(dts, [&](int s) { return p.dtv[k.chan(s)]; });
  if (FWD) {
    k.own(lams, [&](int s) { return p.lamv[k.chan(s)]; });
    k.own(xs, [&](int s) { return to_f32(X[(k.row0 + s) * p.D + k.d]); });
    if (k.ts > 0) px = to_f32(X[(k.row0 - 1) * p.D + k.d]);
  }
  if (DH) k.own(dys, [&](int s) { return to_f32(DY[(k.row0 + s) * p.D + k.d]); });
  k.stage(DH);
#pragma unroll
  for (int u = 0; u < UN; ++u) phi[u] = k.two(p.ck_phi + k.wrow() * p.Kp, u);
  k.rates(A);
  __syncthreads();
  f2 h[PR], pb[PR];
  if (FWD) {
#pragma unroll
    for (int r = 0; r < PR; ++r) h[r] = 0ull;
    k.before(phi, pb);
  }
#pragma unroll
  for (int s = 0; s < W; ++s) {
    const float dt = k.of(dts, s);
    f2 gx = 0ull, bx = 0ull;
    if (FWD) {
      const float lam = k.of(lams, s), x = k.of(xs, s);
      gx = dup2(lam * dt * x);
      bx = dup2((1.f - lam) * dt * px);
      px = x;
    }
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      f2 sn, cs;
      phi[u] = wrap2(mad2(dup2(dt), th[s][u], phi[u]));
      sincos2(phi[u], sn, cs);
      const f2 al0 = decay2(A[2 * u], dup2(dt)), al1 = decay2(A[2 * u + 1], dup2(dt));
      if (DH) {
        slot(s, 2 * u) = al0;
        slot(s, 2 * u + 1) = al1;
        slot(s, PR + 2 * u) = sn;
        slot(s, PR + 2 * u + 1) = cs;
      }
      if (FWD) {
        f2 b0, b1;
        k.rot_b(s, u, sn, cs, b0, b1);
        h[2 * u] = mad2(al0, mad2(bx, pb[2 * u], h[2 * u]), mul2(gx, b0));
        h[2 * u + 1] = mad2(al1, mad2(bx, pb[2 * u + 1], h[2 * u + 1]), mul2(gx, b1));
        pb[2 * u] = b0;
        pb[2 * u + 1] = b1;
      }
    }
  }
  if (FWD) {
#pragma unroll
    for (int u = 0; u < UN; ++u) k.put_states(p.ck_h + k.wrow() * p.N, u, h[2 * u], h[2 * u + 1]);
  }
  if (DH) {
    f2 dh[PR];
#pragma unroll
    for (int r = 0; r < PR; ++r) dh[r] = 0ull;
#pragma unroll
    for (int s = W - 1; s >= 0; --s) {
      const f2 dy = dup2(k.of(dys, s));
#pragma unroll
      for (int u = 0; u < UN; ++u) {
        f2 c0, c1;
        k.rot_c(s, u, slot(s, PR + 2 * u), slot(s, PR + 2 * u + 1), c0, c1);
        dh[2 * u] = mul2(slot(s, 2 * u), mad2(dy, c0, dh[2 * u]));
        dh[2 * u + 1] = mul2(slot(s, 2 * u + 1), mad2(dy, c1, dh[2 * u + 1]));
      }
    }
#pragma unroll
    for (int u = 0; u < UN; ++u) k.put_states(p.dhk + k.wrow() * p.N, u, dh[2 * u], dh[2 * u + 1]);
  }
}

// ------------------------------------------------------------ forward walk
template <typename IO, int PR, int LPC, bool PLAIN>
__global__ void __launch_bounds__(256) m3w_out_kernel(M3P p) {
  begin_dependent();
  using K = Walker<IO, PR, LPC, PLAIN>;
  constexpr int UN = K::UN;
  extern __shared__ f2 hist[];
  const K k(p, reinterpret_cast<float*>(hist));
  const IO* X = static_cast<const IO*>(p.x);
  IO* Y = static_cast<IO*>(p.y);
  f2 th[W][UN], h[PR], phi[UN], pb[PR], A[PR];
  k.thetas(th);
  float dts[K::OWN], lams[K::OWN], xs[K::OWN];
  k.own(dts, [&](int s) { return p.dtv[k.chan(s)]; });
  k.own(lams, [&](int s) { return p.lamv[k.chan(s)]; });
  k.own(xs, [&](int s) { return to_f32(X[(k.row0 + s) * p.D + k.d]); });
  float px = k.ts > 0 ? to_f32(X[(k.row0 - 1) * p.D + k.d]) : 0.f;
  k.stage(true);
#pragma unroll
  for (int u = 0; u < UN; ++u) {
    phi[u] = k.two(p.ck_phi + k.wrow() * p.Kp, u);
    k.states(p.ck_h + k.wrow() * p.N, u, h[2 * u], h[2 * u + 1]);
  }
  k.rates(A);
  __syncthreads();
  k.before(phi, pb);
  float ys[K::OWN];
#pragma unroll
  for (int s = 0; s < W; ++s) {
    const float dt = k.of(dts, s), lam = k.of(lams, s), x = k.of(xs, s);
    const f2 gx = dup2(lam * dt * x), bx = dup2((1.f - lam) * dt * px);
    px = x;
    f2 part = 0ull;
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      f2 sn, cs, b0, b1, c0, c1;
      phi[u] = wrap2(mad2(dup2(dt), th[s][u], phi[u]));
      sincos2(phi[u], sn, cs);
      k.rot_b(s, u, sn, cs, b0, b1);
      k.rot_c(s, u, sn, cs, c0, c1);
      h[2 * u] = mad2(decay2(A[2 * u], dup2(dt)), mad2(bx, pb[2 * u], h[2 * u]), mul2(gx, b0));
      h[2 * u + 1] = mad2(decay2(A[2 * u + 1], dup2(dt)), mad2(bx, pb[2 * u + 1], h[2 * u + 1]), mul2(gx, b1));
      part = mad2(h[2 * u], c0, part);
      part = mad2(h[2 * u + 1], c1, part);
      pb[2 * u] = b0;
      pb[2 * u + 1] = b1;
    }
    const float y = group_sum<LPC>(sum2(part));
    if (k.sl == s % LPC) ys[s / LPC] = y;
  }
#pragma unroll
  for (int o = 0; o < K::OWN; ++o) {
    const int s = k.sl + LPC * o;
    if (s < W && k.in(s)) Y[(k.row0 + s) * p.D + k.d] = from_f32<IO>(ys[o]);
  }
}

// ----------------------------------------------------------- backward walk
// Sums of N = 4 PR values over the channels of a warp: each exchange halves the values a lane still carries, the
// channel's bit choosing the half it keeps.  On return v[0 .. N / CPW) of channel c are the sums of the values first ..
template <int N, int CPW, int LPC>
__device__ __forceinline__ int sum_channels(float (&v)[N], int ch) {
  int first = 0;
#pragma unroll
  for (int m = CPW / 2, n = N / 2; m > 0; m /= 2, n /= 2) {
    const bool up = (ch & m) != 0;
#pragma unroll
    for (int x = 0; x < n; ++x) {
      const float send = up ? v[x] : v[x + n], keep = up ? v[x + n] : v[x];
      v[x] = keep + __shfl_xor_sync(0xffffffffu, send, m * LPC);
    }
    if (up) first += n;
  }
  return first;
}
// Sums of four values over the lanes of a channel: lane sl ends up with that of value sl & 3.
template <int LPC>
__device__ __forceinline__ float sum_lanes4(float a, float b, float c, float d, int sl) {
  const bool b0 = sl & 1, b1 = sl & 2;
  const float u0 = (b0 ? b : a) + __shfl_xor_sync(0xffffffffu, b0 ? a : b, 1);
  const float u1 = (b0 ? d : c) + __shfl_xor_sync(0xffffffffu, b0 ? c : d, 1);
  float v = (b1 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b1 ? u0 : u1, 2);
#pragma unroll
  for (int o = 4; o < LPC; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int PR, int LPC>
struct GradSmem {  // bytes per thread and per warp
  static constexpr int kThread = W * 2 * PR * 8, kWarp = W * 2 * 2 * PR * LPC * 4 + W * (32 / LPC) * 5 * 4;
};
// grid (D / channels of a CTA, windows, B).  What a step needs of its channel waits in shared memory, one read for all lanes (four
// shuffles and the products of three scalars a step and pass before), and its results take the place; the decay is computed again
// on the way back.  Of 96 registers (no spills to speak of) a quarter of an SM holds five warps, of 80 six: the fewer where a CTA
// more fits an SM for it and the grid takes a round of CTAs less (launch_grad; CTAs of seven warps alone; 256 x 448 channels with
// 96 registers a call of 39.4 us, 40.4 with 80; 2048 x 448 171 and 164).  4096 x 448 channels of 16 states, seven warps a CTA: 170 us with two CTAs an SM and 96
// registers, 154 with three and 80 (76 bytes spilled).  2 x 1024 x 128 channels, four warps and five CTAs either way: 29.2 with 96
// registers, 30.8 with 80.
template <typename IO, int PR, int LPC, bool PLAIN, int REGS>
__global__ void __maxnreg__(REGS) m3w_grad_kernel(M3P p) {
  begin_dependent();
  using K = Walker<IO, PR, LPC, PLAIN>;
  constexpr int UN = K::UN, CPW = K::CPW, KEEP = 4 * PR / CPW > 0 ? 4 * PR / CPW : 1, NR = 2 * K::NP;
  static_assert(4 * PR >= CPW, "a lane keeps at least one sum");
  extern __shared__ f2 hist[];  // [W][2 PR][threads]: h after the step, sine / cosine
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5;
  float* red = reinterpret_cast<float*>(hist + (size_t)W * 2 * PR * blockDim.x);  // [W][warps][2 (dB, dC)][NR]
  // per (step, channel): dt, lambda dt x, (1 - lambda) dt x of the step before, dy, then b.up, q.v, the rest of d/d dt, dx of the
  // later step; and (1 - lambda) dt, then the angle's gradient
  float4* fin = reinterpret_cast<float4*>(red + (size_t)W * warps * 2 * NR);
  float* fin5 = reinterpret_cast<float*>(fin + W * warps * CPW);
  const K k(p, fin5 + W * warps * CPW);
  auto slot = [&](int s, int x) -> f2& { return hist[(s * (2 * PR) + x) * blockDim.x + threadIdx.x]; };
  const IO *X = static_cast<const IO*>(p.x), *DY = static_cast<const IO*>(p.dy);
  const bool per_head = k.per_head;
  auto at = [&](int s) { return s * warps * CPW + k.wc; };
  f2 th[W][UN], h[PR], pb[PR], phi[UN], dh[PR], pgb[PR], A[PR];
  k.thetas(th);
  float dts[K::OWN], lams[K::OWN], xs[K::OWN], dys[K::OWN];
  k.own(dts, [&](int s) { return p.dtv[k.chan(s)]; });
  k.own(lams, [&](int s) { return p.lamv[k.chan(s)]; });
  k.own(xs, [&](int s) { return to_f32(X[(k.row0 + s) * p.D + k.d]); });
  k.own(dys, [&](int s) { return to_f32(DY[(k.row0 + s) * p.D + k.d]); });
  const float px0 = k.ts > 0 ? to_f32(X[(k.row0 - 1) * p.D + k.d]) : 0.f;
  float xps[K::OWN];  // x of the step before
#pragma unroll
  for (int o = 0; o < K::OWN; ++o) {
    const int s = k.sl + LPC * o;
    const float xp = __shfl_sync(0xffffffffu, o > 0 && k.sl == LPC - 1 ? xs[o > 0 ? o - 1 : 0] : xs[o], (k.sl == 0 ? k.base + LPC - 1 : k.lane - 1));
    xps[o] = s == 0 ? px0 : xp;
    if (s < W) {
      const float bf = (1.f - lams[o]) * dts[o];
      fin[at(s)] = make_float4(dts[o], lams[o] * dts[o] * xs[o], bf * xps[o], dys[o]);
      fin5[at(s)] = bf;
    }
  }
  const float px = k.of(xs, W - 1);
  const bool more = k.in(W);  // a window follows: its first step sends something back to this one's last
  const float bf_e = more ? (1.f - p.lamv[k.chan(W)]) * p.dtv[k.chan(W)] : 0.f;
  k.stage(true);
#pragma unroll
  for (int u = 0; u < UN; ++u) {
    phi[u] = k.two(p.ck_phi + k.wrow() * p.Kp, u);
    k.states(p.ck_h + k.wrow() * p.N, u, h[2 * u], h[2 * u + 1]);
    k.states(p.dhk + k.wrow() * p.N, u, dh[2 * u], dh[2 * u + 1]);
  }
  k.rates(A);
  __syncthreads();
  k.before(phi, pb);
  f2 hs[PR], pbs[PR];  // state and rotated b before the window's first step
#pragma unroll
  for (int r = 0; r < PR; ++r) {
    hs[r] = h[r];
    pbs[r] = pb[r];
  }
  // ---- replay, keeping state, sine and cosine of every step ----
#pragma unroll
  for (int s = 0; s < W; ++s) {
    const float4 f = fin[at(s)];
    const f2 dt = dup2(f.x), gx = dup2(f.y), bx = dup2(f.z);
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      f2 sn, cs, b0, b1;
      phi[u] = wrap2(mad2(dt, th[s][u], phi[u]));
      sincos2(phi[u], sn, cs);
      k.rot_b(s, u, sn, cs, b0, b1);
      const f2 al0 = decay2(A[2 * u], dt), al1 = decay2(A[2 * u + 1], dt);
      h[2 * u] = mad2(al0, mad2(bx, pb[2 * u], h[2 * u]), mul2(gx, b0));
      h[2 * u + 1] = mad2(al1, mad2(bx, pb[2 * u + 1], h[2 * u + 1]), mul2(gx, b1));
      pb[2 * u] = b0;
      pb[2 * u + 1] = b1;
      slot(s, 2 * u) = h[2 * u];
      slot(s, 2 * u + 1) = h[2 * u + 1];
      slot(s, PR + 2 * u) = sn;
      slot(s, PR + 2 * u + 1) = cs;
    }
  }
  // ---- what the first step of the next window sends back: its decayed `up` is the dh that enters here ----
  f2 dal[PR], carry[UN];
  f2 pend = 0ull;  // contribution of step t+1 to dx_t (lane partial)
#pragma unroll
  for (int u = 0; u < UN; ++u) {
    carry[u] = 0ull;
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const int r = 2 * u + y;
      const f2 v = mul2(dup2(bf_e), dh[r]);
      dal[r] = 0ull;
      pend = mad2(pb[r], v, pend);
      pgb[r] = mul2(dup2(px), v);
    }
  }
  // ---- reverse: pb = rotated b of the step, q = that of the step before ----
#pragma unroll
  for (int s = W - 1; s >= 0; --s) {
    const float4 f = fin[at(s)];
    const float bf = fin5[at(s)];
    const f2 dt2 = dup2(f.x), gx = dup2(f.y), bx = dup2(f.z), dy2 = dup2(f.w);
    f2 s_bu = 0ull, s_qv = 0ull, s_a = 0ull, s_w = 0ull, s_ca = 0ull;
    float rows[4 * PR];  // this lane's values of dB (first half) and dC of the step
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const f2 sn = slot(s, PR + 2 * u), cs = slot(s, PR + 2 * u + 1), nsn = neg2(sn);
      f2 q[2], c[2], gb[2], gc[2];
      if (s > 0) k.rot_b(s - 1, u, slot(s - 1, PR + 2 * u), slot(s - 1, PR + 2 * u + 1), q[0], q[1]);
      else { q[0] = pbs[2 * u]; q[1] = pbs[2 * u + 1]; }
      k.rot_c(s, u, sn, cs, c[0], c[1]);
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int r = 2 * u + y;
        const f2 hb = s > 0 ? slot(s - 1, r) : hs[r];
        const f2 up = mad2(dy2, c[y], dh[r]);
        const f2 v = mul2(decay2(A[r], dt2), up);
        s_bu = mad2(pb[r], up, s_bu);
        s_qv = mad2(q[y], v, s_qv);
        gb[y] = mad2(gx, up, pgb[r]);
        gc[y] = mul2(dy2, slot(s, r));
        const f2 wv = mul2(A[r], mul2(v, mad2(bx, q[y], hb)));
        s_w = add2(s_w, wv);
        dal[r] = mad2(dt2, wv, dal[r]);
        pgb[r] = mul2(bx, v);
        dh[r] = v;
      }
      // rotation adjoint: rows of dB and dC, and the angle gradient of the pairs
      const float2 be = unpack2(mad2(nsn, gb[1], mul2(cs, gb[0]))), bo = unpack2(mad2(sn, gb[0], mul2(cs, gb[1])));
      const float2 ce = unpack2(mad2(nsn, gc[1], mul2(cs, gc[0]))), co = unpack2(mad2(sn, gc[0], mul2(cs, gc[1])));
      float* rb = rows + 4 * u;
      float* rc = rows + 2 * PR + 4 * u;
      rb[0] = be.x; rb[1] = bo.x; rb[2] = be.y; rb[3] = bo.y;
      rc[0] = ce.x; rc[1] = co.x; rc[2] = ce.y; rc[3] = co.y;
      f2 turn = mad2(pb[2 * u + 1], gb[0], mul2(c[1], gc[0]));
      turn = add2(turn, neg2(mad2(pb[2 * u], gb[1], mul2(c[0], gc[1]))));
      carry[u] = add2(carry[u], turn);
      pb[2 * u] = q[0];
      pb[2 * u + 1] = q[1];
      s_a = mad2(carry[u], th[s][u], s_a);
      if (per_head) s_ca = add2(s_ca, carry[u]);
      else if (k.in(s)) k.put_two(p.dtheta + ((k.row0 + s) * p.D + k.d) * p.Kp, u, mul2(carry[u], dt2));
    }
    s_a = add2(s_a, s_w);
    const float v = sum_lanes4<LPC>(sum2(s_bu), sum2(s_qv), sum2(s_a), sum2(pend), k.sl);
    __syncwarp();
    if (k.sl < 4) reinterpret_cast<float*>(fin + at(s))[k.sl] = v;
    if (per_head) {
      const float t = group_sum<LPC>(sum2(s_ca));
      if (k.sl == 0) fin5[at(s)] = t;
    }
    pend = mul2(dup2(bf), s_qv);
    const int first = sum_channels<4 * PR, CPW, LPC>(rows, k.lane / LPC);
    float* dst = red + (size_t)(s * warps + warp) * 2 * NR;
#pragma unroll
    for (int y = 0; y < KEEP; ++y) {
      const int v2 = first + y;  // value of this lane: dB for v2 < 2 PR, then dC
      dst[(v2 >= 2 * PR ? NR : 0) + k.sl * 2 * PR + v2 % (2 * PR)] = rows[y];
    }
  }
#pragma unroll
  for (int u = 0; u < UN; ++u) k.put_two(p.ang + k.wrow() * p.Kp, u, carry[u]);
  // da_log: d/d a_log = d/dA * A  (A = -exp(a_log)); the closed form above already carries A
  if (per_head) {
    f2 sum = 0ull;
#pragma unroll
    for (int r = 0; r < PR; ++r) sum = add2(sum, dal[r]);
    const float v = group_sum<LPC>(sum2(sum));
    if (k.sl == 0) p.dal_part[k.wrow()] = v;
  } else {
#pragma unroll
    for (int u = 0; u < UN; ++u) k.put_states(p.dal_part + k.wrow() * p.N, u, dal[2 * u], dal[2 * u + 1]);
  }
  __syncwarp();
#pragma unroll
  for (int o = 0; o < K::OWN; ++o) {  // the lane that owns a step finishes its scalars: dx, ddt, dlambda
    const int s = k.sl + LPC * o;
    if (s < W && k.in(s)) {
      const float4 f = fin[at(s)];  // b.up, q.v, rest, dx of later step
      const float dt = dts[o], lam = lams[o], x = xs[o], xprev = xps[o];
      const size_t i = (k.row0 + s) * p.D + k.d, ci = k.chan(s);
      static_cast<IO*>(p.dx)[i] = from_f32<IO>(fmaf(lam * dt, f.x, f.w));
      const float dsp = (f.z + (1.f - lam) * xprev * f.y + lam * x * f.x) * m3_sigmoid(p.dt[ci]);
      const float dlam = dt * (x * f.x - xprev * f.y) * lam * (1.f - lam);
      if (per_head) {  // per channel; m3_head_sum_kernel adds the channels of a head
        const size_t btd = (size_t)p.B * p.T * p.D;
        p.hd[i] = dsp;
        p.hd[btd + i] = dlam;
        p.hd[2 * btd + i] = fin5[at(s)] * dt;
      } else {
        p.ddt[ci] = dsp;
        p.dlam[ci] = dlam;
      }
    }
  }
  __syncthreads();
  const int g = k.d / k.ix.cpg, slice = (k.d % k.ix.cpg) / (warps * CPW), steps = min(W, p.T - k.ts);
  for (int i = threadIdx.x; i < steps * 2 * p.N; i += blockDim.x) {
    const int s = i / (2 * p.N), v = i - s * 2 * p.N, which = v >= p.N, n = v - which * p.N;
    const float* src = red + (size_t)s * warps * 2 * NR + which * NR + n;
    float acc = 0.f;
    for (int y = 0; y < warps; ++y) acc += src[(size_t)y * 2 * NR];
    (which ? p.pc32 : p.pb32)[(((k.row0 + s) * p.G + g) * p.S + slice) * p.N + n] = acc;
  }
}

// The angle gradient reaches every earlier step: the later windows' sums are added to ddt and dtheta of each step
// (the walks used only the sums inside their own window).
template <typename IO, int PR, int LPC, bool PLAIN>
__global__ void __launch_bounds__(256) m3w_fix_kernel(M3P p) {
  begin_dependent();
  using K = Walker<IO, PR, LPC, PLAIN>;
  constexpr int UN = K::UN;
  const K k(p, nullptr);
  if (k.w == p.nW - 1) return;  // nothing comes after the last window (every other one is whole)
  const bool per_head = k.per_head;
  const size_t stride = (size_t)p.D * p.Kp;
  float* dst = p.dtheta + (k.row0 * p.D + k.d) * p.Kp;
  f2 off[UN], th[W][UN], dth[W][UN];
#pragma unroll
  for (int u = 0; u < UN; ++u) off[u] = k.two(p.ang + k.wrow() * p.Kp, u);
  k.thetas(th);
  if (!per_head) {
#pragma unroll
    for (int s = 0; s < W; ++s)
#pragma unroll
      for (int u = 0; u < UN; ++u) dth[s][u] = k.two(dst + s * stride, u);
  }
  float dts[K::OWN], raw[K::OWN], add[K::OWN];
  k.own(dts, [&](int s) { return p.dtv[k.chan(s)]; });
  k.own(raw, [&](int s) { return p.dt[k.chan(s)]; });
#pragma unroll
  for (int s = 0; s < W; ++s) {
    const f2 dt = dup2(k.of(dts, s));
    f2 acc = 0ull;
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      acc = mad2(off[u], th[s][u], acc);
      if (!per_head) k.put_two(dst + s * stride, u, mad2(off[u], dt, dth[s][u]));
    }
    const float v = group_sum<LPC>(sum2(acc));
    if (k.sl == s % LPC) add[s / LPC] = v;
  }
  float o = 0.f;
  if (per_head) {
    f2 sum = 0ull;
#pragma unroll
    for (int u = 0; u < UN; ++u) sum = add2(sum, off[u]);
    o = group_sum<LPC>(sum2(sum));
  }
#pragma unroll
  for (int x = 0; x < K::OWN; ++x) {
    const int s = k.sl + LPC * x;
    if (s < W) {
      const float dsp = add[x] * m3_sigmoid(raw[x]);
      if (per_head) {
        const size_t btd = (size_t)p.B * p.T * p.D, i = (k.row0 + s) * p.D + k.d;
        p.hd[i] += dsp;
        p.hd[2 * btd + i] += o * dts[x];
      } else {
        p.ddt[k.chan(s)] += dsp;
      }
    }
  }
}
}  // namespace m3w

// --------------------------------------------------------------------- host
using namespace m3w;

// Lanes per channel: two pairs per lane (four beyond 64 pairs), at least four lanes; a warp's channels share a group.
M3WinShape m3w_shape(const M3P& p) {
  const int pr = p.Kp > 64 ? 4 : 2;
  M3WinShape s{4, 1};
  while (s.lanes < 32 && (s.lanes * pr < p.Kp || p.D / p.G % (32 / s.lanes) != 0)) s.lanes *= 2;
  const int per_group = p.D / p.G / (32 / s.lanes), cap = pr == 4 ? 4 : 8;
  for (int w = 1; w <= cap; ++w)
    if (per_group % w == 0) s.warps = w;
  return s;
}

#define M3W_DISPATCH(lanes, p, call)                                                                      \
  do {                                                                                                    \
    const bool plain = (p).vec && (p).NH == 0;                                                            \
    if ((p).Kp > 64) { constexpr int PRV = 4, LPCV = 32; constexpr bool PL = false; call; }               \
    else if ((lanes) == 4) {                                                                              \
      constexpr int PRV = 2, LPCV = 4;                                                                    \
      if (plain) { constexpr bool PL = true; call; } else { constexpr bool PL = false; call; }            \
    } else if ((lanes) == 8) {                                                                            \
      constexpr int PRV = 2, LPCV = 8;                                                                    \
      if (plain) { constexpr bool PL = true; call; } else { constexpr bool PL = false; call; }            \
    }                                                                                                     \
    else if ((lanes) == 16) { constexpr int PRV = 2, LPCV = 16; constexpr bool PL = false; call; }        \
    else { constexpr int PRV = 2, LPCV = 32; constexpr bool PL = false; call; }                           \
  } while (0)

struct M3WGrid {
  M3WinShape shape;
  int threads;
};
static M3WGrid m3w_grid(const M3P& p) {
  const M3WinShape s = m3w_shape(p);
  return {s, 32 * s.warps};
}
// A walk over every window: launch(parameters, grid), once per 65535 windows (a grid axis).
template <typename F>
static void m3w_walk(const M3P& p, const M3WGrid& g, F&& launch) {
  const int channels = g.shape.warps * (32 / g.shape.lanes);
  for (M3P q = p; q.w0 < p.nW; q.w0 += 65535) launch(q, dim3((p.D + channels - 1) / channels, std::min(65535, p.nW - q.w0), p.B));
}
static dim3 chain_grid(const M3P& p, int chains, int kinds) { return dim3((chains + kChains - 1) / kChains, p.B, kinds); }
// Windows of a segment: as many as a sequence fills, up to 16 (registers).
template <typename F>
static void by_segment(const M3P& p, F&& f) {
  if (p.nW <= 4 * kSegs) f(std::integral_constant<int, 4>{});
  else if (p.nW <= 8 * kSegs) f(std::integral_constant<int, 8>{});
  else f(std::integral_constant<int, 16>{});
}

template <typename IO, int PR, int LPC, bool PLAIN, bool FWD, bool DH>
static mxb_status launch_local(const M3P& p, const M3WGrid& g, cudaStream_t st) {
  constexpr int per_thread = DH ? W * 2 * PR * 8 : 0, rows = kRowBytes<PR, LPC>;
  const int sm = per_thread * g.threads + rows;
  if (MXB_ALLOW_SMEM(per_thread * (PR == 4 ? 128 : 256) + rows, m3w_local_kernel<IO, PR, LPC, PLAIN, FWD, DH>) != MXB_OK) return MXB_ERR_CUDA;
  m3w_walk(p, g, [&](const M3P& q, dim3 grid) {
    MXB_LAUNCH("m3w_local_kernel", st, (launch_kernel(m3w_local_kernel<IO, PR, LPC, PLAIN, FWD, DH>, grid, g.threads, sm, st, q)));
  });
  return MXB_OK;
}
template <typename IO, int PR, int LPC, bool PLAIN>
static mxb_status launch_grad(const M3P& p, const M3WGrid& g, cudaStream_t st) {
  constexpr int per_warp = 32 * GradSmem<PR, LPC>::kThread + GradSmem<PR, LPC>::kWarp, rows = kRowBytes<PR, LPC>;
  const int sm = g.shape.warps * per_warp + rows;
  auto launch = [&](auto regs) {
    constexpr int REGS = decltype(regs)::value;
    if (MXB_ALLOW_SMEM((PR == 4 ? 4 : 8) * per_warp + rows, m3w_grad_kernel<IO, PR, LPC, PLAIN, REGS>) != MXB_OK) return MXB_ERR_CUDA;
    m3w_walk(p, g, [&](const M3P& q, dim3 grid) {
      MXB_LAUNCH("m3w_grad_kernel", st, (launch_kernel(m3w_grad_kernel<IO, PR, LPC, PLAIN, REGS>, grid, g.threads, sm, st, q)));
    });
    return MXB_OK;
  };
  if constexpr (PR == 4) {
    return launch(std::integral_constant<int, 255>{});  // (shared memory leaves one CTA of four warps an SM)
  } else {
    if constexpr (LPC == 4) {  // (no other lane count has a number of warps for which it matters)
      const size_t grid = (size_t)p.D / (g.shape.warps * 8) * p.nW * p.B;
      auto rounds = [&](int warps) {  // of CTAs over the GPU, where an SM's registers hold so many warps
        const size_t at_once = 148 * std::min(warps / g.shape.warps, 228 * 1024 / (sm + 1024));
        return (grid + at_once - 1) / at_once;
      };
      if (rounds(24) < rounds(20)) return launch(std::integral_constant<int, 80>{});
    }
    return launch(std::integral_constant<int, 96>{});
  }
}
template <typename IO>
static mxb_status prepare(const M3P& p, const M3WGrid& g, cudaStream_t st) {
  m3w_walk(p, g, [&](const M3P& q, dim3 grid) {
    M3W_DISPATCH(g.shape.lanes, p, MXB_LAUNCH("m3w_prepare_kernel", st, (launch_kernel(m3w_prepare_kernel<IO, PRV, LPCV, PL>, grid, g.threads, 0, st, q))));
  });
  by_segment(p, [&](auto per) {
    MXB_LAUNCH("m3w_phase_scan_kernel", st,
               (launch_kernel(m3w_phase_scan_kernel<decltype(per)::value>, chain_grid(p, p.D * p.Kp, 1), kScanThreads, 0, st, p)));
  });
  return check_launch("mamba3 window preparation");
}

static void linear_scan(const M3P& p, int first, int kinds, cudaStream_t st) {
  by_segment(p, [&](auto per) {
    MXB_LAUNCH("m3w_linear_scan_kernel", st,
               (launch_kernel(m3w_linear_scan_kernel<decltype(per)::value>, chain_grid(p, p.D * p.N, kinds), kScanThreads, 0, st, p, first)));
  });
}

template <typename IO>
static mxb_status forward(const M3P& p, cudaStream_t st) {
  const M3WGrid g = m3w_grid(p);
  mxb_status s = prepare<IO>(p, g, st);
  if (s != MXB_OK) return s;
  M3W_DISPATCH(g.shape.lanes, p, (s = launch_local<IO, PRV, LPCV, PL, true, false>(p, g, st)));
  if (s != MXB_OK) return s;
  linear_scan(p, 0, 1, st);
  m3w_walk(p, g, [&](const M3P& q, dim3 grid) {
    M3W_DISPATCH(g.shape.lanes, p, MXB_LAUNCH("m3w_out_kernel", st, (launch_kernel(m3w_out_kernel<IO, PRV, LPCV, PL>, grid, g.threads, kRowBytes<PRV, LPCV>, st, q))));
  });
  return check_launch("mamba3 window-parallel forward");
}
// have_states: angles and states at the window starts (and dtv, lamv) are those a forward on the same inputs left.
template <typename IO>
static mxb_status backward(const M3P& p, bool have_states, cudaStream_t st) {
  const M3WGrid g = m3w_grid(p);
  mxb_status s = MXB_OK;
  if (have_states) {
    M3W_DISPATCH(g.shape.lanes, p, (s = launch_local<IO, PRV, LPCV, PL, false, true>(p, g, st)));
  } else {
    s = prepare<IO>(p, g, st);
    if (s == MXB_OK) M3W_DISPATCH(g.shape.lanes, p, (s = launch_local<IO, PRV, LPCV, PL, true, true>(p, g, st)));
  }
  if (s != MXB_OK) return s;
  const int first = have_states ? 1 : 0;
  linear_scan(p, first, 2 - first, st);
  M3W_DISPATCH(g.shape.lanes, p, (s = launch_grad<IO, PRV, LPCV, PL>(p, g, st)));
  if (s != MXB_OK) return s;
  const int scans = chain_grid(p, p.D * p.Kp, 1).x * p.B, dalogs = m3_dalog_blocks(p);
  by_segment(p, [&](auto per) {
    MXB_LAUNCH("m3w_sums_kernel", st,
               (launch_kernel(m3w_sums_kernel<IO, decltype(per)::value>, scans + dalogs + m3_bc_sum_blocks(p, kScanThreads), kScanThreads, 0,
                              st, p, scans, dalogs)));
  });
  m3w_walk(p, g, [&](const M3P& q, dim3 grid) {
    M3W_DISPATCH(g.shape.lanes, p, MXB_LAUNCH("m3w_fix_kernel", st, (launch_kernel(m3w_fix_kernel<IO, PRV, LPCV, PL>, grid, g.threads, 0, st, q))));
  });
  return check_launch("mamba3 window-parallel backward");
}

mxb_status m3w_sincos_selftest(const float* x, size_t n, float* sn, float* cs, cudaStream_t st) {
  const int grid = (int)std::min<size_t>((n + 511) / 512, 148 * 8);
  MXB_LAUNCH("m3w_sincos_kernel", st, (launch_kernel(m3w_sincos_kernel, grid, 256, 0, st, x, n, sn, cs)));
  return check_launch("m3w_sincos_kernel");
}
mxb_status m3w_forward(const M3P& p, bool f32, cudaStream_t st) {
  return f32 ? forward<float>(p, st) : forward<__nv_bfloat16>(p, st);
}
mxb_status m3w_backward(const M3P& p, bool f32, bool have_states, cudaStream_t st) {
  return f32 ? backward<float>(p, have_states, st) : backward<__nv_bfloat16>(p, have_states, st);
}

}  // namespace mxb
