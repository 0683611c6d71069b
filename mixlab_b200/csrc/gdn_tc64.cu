// Gated delta rule - tensor-core kernels for heads of 64 columns (Dk = Dv = 64), bf16 I/O, fp32 state, chunk 64.
//
// The mathematics of gdn_tc.cu / gdn_tc_bwd.cu on tiles of their true width: half the bytes and a quarter of the state
// of the 128-wide tiles these heads used to ride on, so that two CTAs of the sequential passes (three of the chunk
// backward) share an SM.  What changes beside the sizes:
//
//   A 128-row instruction takes two 64-row products that share their second operand:
//     forward   [w; q] S            and [k^T diag(r); P] v_new  (one operand of 128 columns contracted over its rows: the
//                                   k tile and, behind it, the image of P^T)
//     backward  [P^T; (d q)^T] dO   (the P image and, behind it, the q tile), then  - w^T dv_new  on the lower half alone
//   so that the halves land in TMEM lanes 0-63 and 64-127 and every lane of a warp owns a row.  Where only one half is
//   wanted the other one reads whatever lies beside the operand and its result is not looked at.
//
//   Chunk backward: S0 and dS have buffers of their own, so that z and v_new dS^T share a batch and DQ is formed at the
//   end: five batches instead of six and 128 TMEM columns.
//
// Every kernel is fed by the copy engine.
#include <cstring>

#include "gdn_tc.cuh"

namespace mxb {
namespace g64 {
constexpr int W = 64;          // width of every tile
constexpr int kTile = 8192;    // bytes of a [64][64] bf16 tile

// byte offset of unit (r, c8) of a swizzled tile (one slab)
__device__ __forceinline__ uint32_t sw_unit(int r, int c8) { return (uint32_t)r * 128u + (uint32_t)((c8 ^ (r & 7)) << 4); }

// Rows of a swizzled tile scaled in place by all 256 threads.
__device__ __forceinline__ void scale_rows(uint8_t* tile, const float* s, int nt) {
  for (int u = threadIdx.x; u < 512; u += nt) {
    uint4* unit = reinterpret_cast<uint4*>(tile + 16 * u);  // unit u lies in row u / 8, whatever its column
    *unit = tc::scale_bf16x8(*unit, s[u >> 3]);
  }
}

// ------------------------------------------------------------------ prep
// A chain of dependent steps (prep kernel of gdn_tc.cu); six CTAs per SM overlap theirs (64 TMEM columns, 36 KB).  [k;q]
// (swizzled boxes) -> the P^T image, then v, then u over q, w over k; the fp32 matrix holds A, T and, once it is dead, the
// bf16 T image and T diag(beta).
constexpr int kPrepSmem = 2 * kTile + C * LDA * 4 + 3 * C * 4 + 64 + 1024;
static_assert(6 * (kPrepSmem + 1024) <= 228 * 1024, "six CTAs per SM");

__global__ void __launch_bounds__(128, 6) gdn_tc_prep_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Xk = sm;             // k, then d k, then the w image
  uint8_t* Xq = Xk + kTile;     // q, then the P^T image, then v, then the u image
  uint8_t* Xpt = Xq;
  float* Am = reinterpret_cast<float*>(Xq + kTile);  // [64][LDA]  A, then T in place
  uint8_t* Tt = reinterpret_cast<uint8_t*>(Am);       // T image
  uint8_t* Tb = Tt + kTile;                           // T diag(beta)
  float* gam = Am + C * LDA;
  float* bet = gam + C;
  float* dd = bet + C;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(dd + C);  // [0] MMA, [1] k and q landed, [2] v landed
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H, t0 = c * C;
  const size_t ci = (size_t)bh * p.n + c;
  auto row = [&](int i) { return ((size_t)(b * p.T + t0 + i) * p.H + h); };
  const int imax = min(C, p.T - t0);

  // The first CTA clears the status header: whoever raises it has waited in vain for far longer than this takes.
  if (c == 0 && bh == 0 && tid < 64) p.status[tid] = 0;
  if (tid == 64) {
    for (int m = 0; m < 3; ++m) tc::mbar_init(&mbar[m], 1);
    tc::mbar_fence_init();
    tc::mbar_expect_tx(&mbar[1], 2 * kTile);
    tc::tma_load_4d(tc::smem_u32(Xk), &maps.k, 0, h, t0, b, &mbar[1]);
    tc::tma_load_4d(tc::smem_u32(Xq), &maps.q, 0, h, t0, b, &mbar[1]);
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, 64);
    tc::tmem_relinquish();
  }
  if (warp == 1) {  // in-chunk inclusive cumulative sum of the log gate: two elements per lane
    const bool ok0 = 2 * lane < imax, ok1 = 2 * lane + 1 < imax;
    const float g0 = ok0 ? log_gate_tc(p.gate[row(2 * lane)], p.gate_is_log) : 0.f;
    const float g1 = ok1 ? log_gate_tc(p.gate[row(2 * lane + 1)], p.gate_is_log) : 0.f;
    const float b0 = ok0 ? p.beta[row(2 * lane)] : 0.f, b1 = ok1 ? p.beta[row(2 * lane + 1)] : 0.f;
    float s = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    const float c1 = s, c0 = s - g1;
    gam[2 * lane] = c0; gam[2 * lane + 1] = c1;
    bet[2 * lane] = b0; bet[2 * lane + 1] = b1;
    dd[2 * lane] = exp_nonpos(c0); dd[2 * lane + 1] = exp_nonpos(c1);
    *reinterpret_cast<float2*>(p.gam + ci * C + 2 * lane) = make_float2(c0, c1);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  bool ok = tc::mbar_wait(&mbar[1], 0);
  // D0[128 x 64] = [k;q] k^T
  if (ok && tid == 0) {
    tc::issue_gemm(taddr, tc::kmajor_sw128_tile(Xk, kTile), tc::kmajor_sw128_tile(Xk, kTile), 128, 64, W, false);
    tc::mma_commit(mbar);
  }
  if (ok) ok = tc::mbar_wait(mbar, 0);
  tc::fence_after_sync();
  if (ok) {
    const int i = tid & 63;
    const float gi = gam[i], bi = bet[i];
    for (int c0 = 0; c0 < 64; c0 += 32) {
      float f[32];
      ld_acc32(taddr, warp, c0, f);
      if (tid < 64) {  // A = -(k beta k^T) Gamma, strictly lower (all values before the first store: they overlap)
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) {
          const int j = c0 + jj;
          const float val = -bi * f[jj] * exp_nonpos(gi - gam[j]);
          f[jj] = (j < i) ? val : 0.f;
        }
#pragma unroll
        for (int x = 0; x < 8; ++x)
          *reinterpret_cast<float4*>(Am + i * LDA + c0 + 4 * x) = make_float4(f[4 * x], f[4 * x + 1], f[4 * x + 2], f[4 * x + 3]);
      } else {         // P = (q k^T) Gamma, lower incl. diagonal
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) {
          const int j = c0 + jj;
          const float val = f[jj] * exp_nonpos(gi - gam[j]);
          f[jj] = (j <= i) ? val : 0.f;
        }
        // its transpose for the forward: a warp's 32 rows are 64 consecutive bytes of row j
#pragma unroll
        for (int jj = 0; jj < 32; ++jj)
          *reinterpret_cast<bf16*>(Xpt + sw_unit(c0 + jj, i >> 3) + 2 * (i & 7)) = __float2bfloat16_rn(f[jj]);
        if (p.save) {  // and the image itself for the backward, straight to the workspace
          uint8_t* pimg = reinterpret_cast<uint8_t*>(p.P + ci * C * C);
#pragma unroll
          for (int x = 0; x < 4; ++x) *reinterpret_cast<uint4*>(pimg + sw_unit(i, (c0 >> 3) + x)) = pack8(&f[8 * x]);
        }
      }
    }
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (ok && tid == 96) {  // P^T leaves, then v takes its place (needed long after the solve)
    tc::bulk_store(p.Pt + ci * C * C, tc::smem_u32(Xpt), kTile);
    tc::bulk_commit();
    tc::bulk_wait_read<0>();
    tc::mbar_expect_tx(&mbar[2], kTile);
    tc::tma_load_4d(tc::smem_u32(Xq), &maps.v, 0, h, t0, b, &mbar[2]);
  }
  invert_unit_lower(Am, ok, [&](int t) {  // the other half of the CTA: k <- diag(d) k
    uint4* unit = reinterpret_cast<uint4*>(Xk);
    for (int u = t; u < 512; u += 64) unit[u] = tc::scale_bf16x8(unit[u], dd[u >> 3]);
  });
  {  // the T image and T diag(beta) go over the fp32 matrix: read everything, barrier, write
    uint4 timg[4], tbimg[4];
    load_inverse_images(Am, bet, timg, tbimg);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      sts16(Tt, 16 * (tid + 128 * m), timg[m]);
      sts16(Tb, 16 * (tid + 128 * m), tbimg[m]);
    }
  }
  if (ok) ok = tc::mbar_wait(&mbar[2], 0);  // v
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // w = (T beta)(d k) and u = (T beta) v, weight-stationary: a thread has a row and half of the columns of both
  if (ok && tid == 0) {
    tc::issue_gemm<true>(taddr, tc::kmajor_tile(Tb, C), tc::mnmajor_sw128_tile(Xk, kTile), 64, W, C, false);
    tc::issue_gemm<true>(taddr + 32, tc::kmajor_tile(Tb, C), tc::mnmajor_sw128_tile(Xq, kTile), 64, W, C, false);
    tc::mma_commit(mbar);
    if (p.save) tc::bulk_store(p.Tm + ci * C * C, tc::smem_u32(Tt), kTile);
    tc::bulk_commit();
  }
  if (ok) ok = tc::mbar_wait(mbar, 1);
  tc::fence_after_sync();
  if (ok) {
    const int ir = 32 * (warp & 1) + lane, c8 = 4 * (warp >> 1);
    float f[32];
    ld_acc32(taddr, warp, 0, f);
#pragma unroll
    for (int x = 0; x < 4; ++x) sts16(Xk, sw_unit(ir, c8 + x), pack8(&f[8 * x]));  // the w image is swizzled, the u image is not
    ld_acc32(taddr + 32, warp, 0, f);
#pragma unroll
    for (int x = 0; x < 4; ++x) sts16(Xq, tc::kmajor_unit(ir, c8 + x, W), pack8(&f[8 * x]));
  } else if (tid == 0) {
    atomicExch(p.status, 1);
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  if (tid == 0) {
    if (ok) {
      tc::bulk_store(p.w + ci * C * W, tc::smem_u32(Xk), kTile);
      tc::bulk_store(p.u + ci * C * W, tc::smem_u32(Xq), kTile);
      tc::bulk_commit();
    }
    tc::bulk_wait_read<0>();  // shared memory must outlive the copies
  }
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 64);
}

// ------------------------------------------------------------ state forward
// One CTA (256 threads, two per SM) per (batch, head).  Row r = 32 (warp % 4) + lane of an accumulator, 32 of its
// columns (half warp / 4): rows 0-63 make v_new and own the state, rows 64-127 make the output.  Every operand tile
// is double-buffered and requested two chunks ahead, as soon as the instruction that last read its buffer is done:
//   A  [w; q]     free after [w;q] S        U  u           free after v_new
//   K  k | P^T    free after the update (k is scaled to diag(r) k in the shadow of [w;q] S)
constexpr int kStateFwdSmem = 2 * 2 * kTile + kTile + 2 * 2 * kTile + kTile + kTile + 2 * kTile + 2 * C * 4 + 128 + 1024;
static_assert(2 * (kStateFwdSmem + 1024) <= 228 * 1024, "two CTAs per SM");

__global__ void __launch_bounds__(256, 2) gdn_tc_state_fwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* A1 = sm;                   // x2 [128][64]: w rows, then q rows (swizzled)
  uint8_t* AK = A1 + 4 * kTile;       // x2 [64][128]: k | P^T (two swizzled slabs)
  uint8_t* Ut = AK + 4 * kTile;       // x2 u image
  uint8_t* Sop = Ut + 2 * kTile;      // [64 kk][64 j] bf16 copy of the state
  uint8_t* Vn = Sop + kTile;          // [64 i][64 j] v_new
  uint8_t* Ot = Vn + kTile;           // output tile on its way out (swizzled)
  float* dd = reinterpret_cast<float*>(Ot + kTile);
  float* rr = dd + C;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(rr + C);  // [0] MMA; per buffer: [1 + buf] A, [3 + buf] U, [5 + buf] K
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 8);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int r = tid & 127, i = r & 63, half = tid >> 7, j0 = 32 * half;
  const bool upper = r >= 64;         // the output half (warp-uniform)
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;

  // issued by threads of the output half's second warps, whose epilogues are the short ones
  auto issue_A = [&](int c) {
    if (c < p.n && tid == 64) {
      const uint32_t dst = tc::smem_u32(A1) + (c & 1) * 2 * kTile;
      uint64_t* mb = &mbar[1 + (c & 1)];
      tc::mbar_expect_tx(mb, 2 * kTile);
      tc::bulk_load(dst, p.w + ((size_t)bh * p.n + c) * C * W, kTile, mb);
      tc::tma_load_4d(dst + kTile, &maps.q, 0, h, c * C, b, mb);
    }
  };
  auto issue_U = [&](int c) {
    if (c < p.n && tid == 64) {
      tc::mbar_expect_tx(&mbar[3 + (c & 1)], kTile);
      tc::bulk_load(tc::smem_u32(Ut) + (c & 1) * kTile, p.u + ((size_t)bh * p.n + c) * C * W, kTile, &mbar[3 + (c & 1)]);
    }
  };
  auto issue_K = [&](int c) {
    if (c < p.n && tid == 96) {
      const uint32_t dst = tc::smem_u32(AK) + (c & 1) * 2 * kTile;
      uint64_t* mb = &mbar[5 + (c & 1)];
      tc::mbar_expect_tx(mb, 2 * kTile);
      tc::tma_load_4d(dst, &maps.k, 0, h, c * C, b, mb);
      tc::bulk_load(dst + kTile, p.Pt + ((size_t)bh * p.n + c) * C * C, kTile, mb);
    }
  };
  if (warp == 0) {
    tc::tmem_alloc(tslot, 128);
    tc::tmem_relinquish();
  }
  if (tid == 32) {
    for (int m = 0; m < 7; ++m) tc::mbar_init(&mbar[m], 1);
    tc::mbar_fence_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  for (int c = 0; c < 2; ++c) {
    issue_A(c);
    issue_U(c);
    issue_K(c);
  }
  float S[32];  // state row i, columns j0 .. j0+31 (lower half only)
  {
    const float4* src = reinterpret_cast<const float4*>(p.h0 + ((size_t)bh * W + i) * W + j0);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const float4 t = p.h0 && !upper ? __ldg(src + x) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[4 * x] = t.x; S[4 * x + 1] = t.y; S[4 * x + 2] = t.z; S[4 * x + 3] = t.w;
    }
  }
  const uint32_t taddr = *tslot;
  uint32_t ph = 0;
  bool ok = true;
  // in-chunk cumulative log decay of the chunk ahead, fetched one chunk early
  float g_nxt = p.gam[(size_t)bh * p.n * C + i], gl_nxt = p.gam[(size_t)bh * p.n * C + C - 1];
  for (int c = 0; c < p.n; ++c) {
    const size_t ci = (size_t)bh * p.n + c;
    const int t0 = c * C, buf = c & 1;
    const uint32_t lph = (c >> 1) & 1;
    uint8_t* A1c = A1 + buf * 2 * kTile;
    uint8_t* AKc = AK + buf * 2 * kTile;
    const float glast = gl_nxt, g = g_nxt;
    if (c + 1 < p.n) {
      g_nxt = p.gam[(ci + 1) * C + i];
      gl_nxt = p.gam[(ci + 1) * C + C - 1];
    }
    const float L = exp_nonpos(glast);
    if (tid < C) rr[tid] = exp_nonpos(glast - g);
    const float di = exp_nonpos(g);
    if (!upper) {
#pragma unroll
      for (int x = 0; x < 4; ++x) sts16(Sop, tc::mnmajor_unit(i, 4 * half + x, W), pack8(&S[8 * x]));
    }
    if (tid == 0) tc::bulk_wait_read<0>();  // the previous chunk's v_new image has left its tile
    if (ok) ok = tc::mbar_wait(&mbar[1 + buf], lph);
    tc::fence_async_smem();
    tc::fence_before_sync();
    ok = __syncthreads_and(ok);  // also makes the verdict of the bounded waits uniform: all threads leave together
    if (!ok) break;
    tc::fence_after_sync();
    if (tid == 0) {  // D1 = [w;q] S
      tc::issue_gemm(taddr, tc::kmajor_sw128_tile(A1c, kTile), tc::mnmajor_tile(Sop, W), 128, W, W, false);
      tc::mma_commit(mbar);
      if (p.save) {
        tc::bulk_store(p.hs + ci * W * W, tc::smem_u32(Sop), kTile);
        tc::bulk_commit();
      }
    }
    if (tid == 96 && c > 0 && !p.out32) {  // the previous chunk's output tile (complete since the barrier above)
      tc::tma_store_4d(&maps.o, tc::smem_u32(Ot), 0, h, t0 - C, b);
      tc::bulk_commit();
    }
    // in the shadow of the product: k <- diag(r) k
    if (ok) ok = tc::mbar_wait(&mbar[5 + buf], lph);
    scale_rows(AKc, rr, 256);
    if (ok) ok = tc::mbar_wait(mbar, ph);
    ph ^= 1;
    tc::fence_after_sync();
    issue_A(c + 2);
    if (ok) ok = tc::mbar_wait(&mbar[3 + buf], lph);
    float f[32];
    if (ok) {
      ld_acc32(taddr, warp, j0, f);
      if (!upper) {  // v_new = u - w S
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          float e[8];
          unpack8(*reinterpret_cast<const uint4*>(Ut + buf * kTile + tc::kmajor_unit(i, 4 * half + x, W)), e);
#pragma unroll
          for (int y = 0; y < 8; ++y) e[y] -= f[8 * x + y];
          sts16(Vn, tc::mnmajor_unit(i, 4 * half + x, W), pack8(e));
        }
      } else {
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) f[jj] *= di;
      }
    }
    if (tid == 0 || tid == 96) tc::bulk_wait_read<0>();  // the state image / the previous output tile has left its tile
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    issue_U(c + 2);
    if (ok && tid == 0) {  // D2 = [k^T diag(r); P] v_new
      tc::issue_gemm(taddr + 64, tc::mnmajor_sw128_tile(AKc, kTile), tc::mnmajor_tile(Vn, W), 128, W, C, false);
      tc::mma_commit(mbar);
      if (p.save) {
        tc::bulk_store(p.vn + ci * C * W, tc::smem_u32(Vn), kTile);
        tc::bulk_commit();
      }
    }
    if (ok) {
      ok = tc::mbar_wait(mbar, ph);
      ph ^= 1;
    }
    tc::fence_after_sync();
    issue_K(c + 2);
    if (ok) {
      float a[32];
      ld_acc32(taddr + 64, warp, j0, a);
      if (upper) {  // out = E(gam)(q S) + P v_new
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) a[jj] += f[jj];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          if (!p.out32) sts16(Ot, sw_unit(i, 4 * half + x), pack8(&a[8 * x]));
          else if (t0 + i < p.T) put_wide(p.out32 + ((size_t)(b * p.T + t0 + i) * p.H + h) * W + j0 + 8 * x, pack8(&a[8 * x]));
        }
      } else {      // S <- E(gam_last) S + (k r)^T v_new
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) S[jj] = fmaf(L, S[jj], a[jj]);
      }
    }
    tc::fence_before_sync();
  }
  tc::fence_async_smem();
  __syncthreads();
  if (ok && tid == 96 && !p.out32) {  // the last chunk's output tile
    tc::tma_store_4d(&maps.o, tc::smem_u32(Ot), 0, h, (p.n - 1) * C, b);
    tc::bulk_commit();
  }
  if (tid == 0 || tid == 96) tc::bulk_wait_read<0>();  // shared memory must outlive the copies
  if (!ok && tid == 0) atomicExch(p.status, 2);
  if (ok && p.hT && !upper) {
    float4* dst = reinterpret_cast<float4*>(p.hT + ((size_t)bh * W + i) * W + j0);
#pragma unroll
    for (int x = 0; x < 8; ++x) dst[x] = make_float4(S[4 * x], S[4 * x + 1], S[4 * x + 2], S[4 * x + 3]);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 128);
}

// ----------------------------------------------------------- state backward
// Reverse over chunks, same shape: rows 0-63 make dv_new = P^T dO + r (k dS), rows 64-127 own dS.
//   A  k, dO, P | q   free after the first batch (q is scaled to diag(E(gam)) q one chunk early)      B  w   free after the second
constexpr int kStateBwdSmem = 3 * kTile + 4 * kTile + 2 * kTile + 2 * kTile + kTile + kTile + 3 * C * 4 + 128 + 1024;
static_assert(2 * (kStateBwdSmem + 1024) <= 228 * 1024, "two CTAs per SM");

__global__ void __launch_bounds__(256, 2) gdn_tc_state_bwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Ak = sm;                   // x2 k (swizzled); the tile behind the second buffer (dSop) is read beside it
  uint8_t* dSop = Ak + 2 * kTile;     // [64 kk][64 j]
  uint8_t* PQ = dSop + kTile;         // x2 [64][128]: P | q (two swizzled slabs)
  uint8_t* dOop = PQ + 4 * kTile;     // x2 dO (swizzled)
  uint8_t* Aw = dOop + 2 * kTile;     // x2 w (swizzled); the tile in front of the first buffer is read beside it
  uint8_t* Bd = Aw + 2 * kTile;       // [64 i][64 j] -dv_new
  float* rr = reinterpret_cast<float*>(Bd + kTile);
  float* ddn = rr + C;                // x2 E(gam) of the chunk whose q is scaled next
  uint64_t* mbar = reinterpret_cast<uint64_t*>(ddn + 2 * C);  // [0] MMA; per buffer: [1 + buf] A, [3 + buf] B
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 8);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int r = tid & 127, i = r & 63, half = tid >> 7, j0 = 32 * half;
  const bool upper = r >= 64;         // the half that owns dS (warp-uniform)
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  auto issue_A = [&](int c) {
    if (c >= 0 && tid == 64) {
      const int o = c & 1;
      uint64_t* mb = &mbar[1 + o];
      tc::mbar_expect_tx(mb, 4 * kTile);
      tc::tma_load_4d(tc::smem_u32(Ak) + o * kTile, &maps.k, 0, h, c * C, b, mb);
      tc::tma_load_4d(tc::smem_u32(dOop) + o * kTile, &maps.dO, 0, h, c * C, b, mb);
      tc::bulk_load(tc::smem_u32(PQ) + o * 2 * kTile, p.P + ((size_t)bh * p.n + c) * C * C, kTile, mb);
      tc::tma_load_4d(tc::smem_u32(PQ) + o * 2 * kTile + kTile, &maps.q, 0, h, c * C, b, mb);
    }
  };
  auto issue_B = [&](int c) {
    if (c >= 0 && tid == 96) {
      tc::mbar_expect_tx(&mbar[3 + (c & 1)], kTile);
      tc::bulk_load(tc::smem_u32(Aw) + (c & 1) * kTile, p.w + ((size_t)bh * p.n + c) * C * W, kTile, &mbar[3 + (c & 1)]);
    }
  };
  if (warp == 0) {
    tc::tmem_alloc(tslot, 128);
    tc::tmem_relinquish();
  }
  if (tid == 32) {
    for (int m = 0; m < 5; ++m) tc::mbar_init(&mbar[m], 1);
    tc::mbar_fence_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  for (int c = p.n - 1; c > p.n - 3; --c) {
    issue_A(c);
    issue_B(c);
  }
  float dS[32];  // row i of dS, columns j0 .. j0+31 (upper half only)
  {
    const float4* src = reinterpret_cast<const float4*>(p.dhT_in + ((size_t)bh * W + i) * W + j0);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const float4 t = p.dhT_in && upper ? __ldg(src + x) : make_float4(0.f, 0.f, 0.f, 0.f);
      dS[4 * x] = t.x; dS[4 * x + 1] = t.y; dS[4 * x + 2] = t.z; dS[4 * x + 3] = t.w;
    }
  }
  const size_t gbase = (size_t)bh * p.n * C;
  float g_cur = p.gam[gbase + (size_t)(p.n - 1) * C + i], gl_cur = p.gam[gbase + (size_t)(p.n - 1) * C + C - 1];
  float g_nxt = 0.f, gl_nxt = 0.f;
  if (p.n > 1) {
    g_nxt = p.gam[gbase + (size_t)(p.n - 2) * C + i];
    gl_nxt = p.gam[gbase + (size_t)(p.n - 2) * C + C - 1];
  }
  if (tid < C) ddn[((p.n - 1) & 1) * C + tid] = exp_nonpos(g_cur);
  __syncthreads();
  const uint32_t taddr = *tslot;
  uint32_t ph = 0;
  // the last chunk's q is scaled here; every later one in the shadow of the previous iteration's second batch
  bool ok = tc::mbar_wait(&mbar[1 + ((p.n - 1) & 1)], 0);
  scale_rows(PQ + ((p.n - 1) & 1) * 2 * kTile + kTile, ddn + ((p.n - 1) & 1) * C, 256);

  for (int c = p.n - 1; c >= 0; --c) {
    const size_t ci = (size_t)bh * p.n + c;
    const int buf = c & 1;
    const uint32_t lph = ((p.n - 1 - c) >> 1) & 1;
    const float glast = gl_cur, g = g_cur;
    g_cur = g_nxt; gl_cur = gl_nxt;
    if (c > 1) {
      g_nxt = p.gam[(ci - 2) * C + i];
      gl_nxt = p.gam[(ci - 2) * C + C - 1];
    }
    const float L = exp_nonpos(glast), ri = exp_nonpos(glast - g);
    if (tid < C && c > 0) ddn[(buf ^ 1) * C + tid] = exp_nonpos(g_cur);  // for the next chunk's q
    if (upper) {
#pragma unroll
      for (int x = 0; x < 4; ++x) sts16(dSop, tc::mnmajor_unit(i, 4 * half + x, W), pack8(&dS[8 * x]));
    }
    if (tid == 0) tc::bulk_wait_read<0>();  // the previous chunk's -dv_new image has left its tile
    tc::fence_async_smem();
    tc::fence_before_sync();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    tc::fence_after_sync();
    if (tid == 0) {
      tc::issue_gemm(taddr, tc::kmajor_sw128_tile(Ak + buf * kTile, kTile), tc::mnmajor_tile(dSop, W), 128, W, W, false);  // k dS
      tc::issue_gemm(taddr + 64, tc::mnmajor_sw128_tile(PQ + buf * 2 * kTile, kTile),
                     tc::mnmajor_sw128_tile(dOop + buf * kTile, kTile), 128, W, C, false);                                 // [P^T; (d q)^T] dO
      tc::mma_commit(mbar);
      tc::bulk_store(p.dhs + ci * W * W, tc::smem_u32(dSop), kTile);
      tc::bulk_commit();
    }
    if (ok) ok = tc::mbar_wait(mbar, ph);
    ph ^= 1;
    tc::fence_after_sync();
    issue_A(c - 2);
    if (ok && !upper) {
      float fa[32], fb[32];
      ld_acc32(taddr, warp, j0, fa);
      ld_acc32(taddr + 64, warp, j0, fb);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float e[8];
#pragma unroll
        for (int y = 0; y < 8; ++y) e[y] = -fmaf(ri, fa[8 * x + y], fb[8 * x + y]);
        sts16(Bd, tc::kmajor_unit(i, 4 * half + x, W), pack8(e));
      }
    }
    if (tid == 0) tc::bulk_wait_read<0>();  // the dS image has left its tile
    if (ok) ok = tc::mbar_wait(&mbar[3 + buf], lph);
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (ok && tid == 0) {  // rows 64-127: ... - w^T dv_new (rows 0-63 have been read)
      tc::issue_gemm(taddr + 64, tc::mnmajor_sw128_tile(Aw + buf * kTile - kTile, kTile), tc::mnmajor_tile(Bd, W), 128, W, C, true);
      tc::mma_commit(mbar);
      tc::bulk_store(p.dvn + ci * C * W, tc::smem_u32(Bd), kTile);
      tc::bulk_commit();
    }
    if (c > 0) {  // in the shadow of the product: the next chunk's q
      if (ok) ok = tc::mbar_wait(&mbar[1 + (buf ^ 1)], ((p.n - c) >> 1) & 1);
      scale_rows(PQ + (buf ^ 1) * 2 * kTile + kTile, ddn + (buf ^ 1) * C, 256);
    }
    if (ok) {
      ok = tc::mbar_wait(mbar, ph);
      ph ^= 1;
    }
    tc::fence_after_sync();
    issue_B(c - 2);
    if (ok && upper) {
      float a[32];
      ld_acc32(taddr + 64, warp, j0, a);
#pragma unroll
      for (int jj = 0; jj < 32; ++jj) dS[jj] = fmaf(L, dS[jj], a[jj]);
    }
    tc::fence_before_sync();
  }
  if (tid == 0) tc::bulk_wait_read<0>();  // shared memory must outlive the copies
  if (!ok && tid == 0) atomicExch(p.status, 3);
  if (ok && p.dh0 && upper) {
    float4* dst = reinterpret_cast<float4*>(p.dh0 + ((size_t)bh * W + i) * W + j0);
#pragma unroll
    for (int x = 0; x < 8; ++x) dst[x] = make_float4(dS[4 * x], dS[4 * x + 1], dS[4 * x + 2], dS[4 * x + 3]);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 128);
}

// ---------------------------------------------------------- chunk backward
// One CTA per chunk, everything that is not the sequential pass (gdn_tc_bwd.cu has the formulas).  Five batches:
//   1  -e = T^T (-dv_new)          dP = dO v_new^T            -> dPG
//   2  z = (-e) S0^T               v_new dS^T                 -> dkp = r (.)     <dS, S0> on the side; (d dO) S0^T
//   3  (-e) v^T                    z k^T                      -> Y;  k k^T
//   4  Y T^T                                                  -> Mb
//   5  dPG^T q + (Mb + Mb^T) k     DQ += dPG k                -> dk, dq
// 128 TMEM columns (weight-stationary products take 32 each) and 75 KB: three CTAs per SM.  A thread has a row and a
// quarter of the columns of every result.  Buffers: dO -> d dO; -dv_new -> -e -> dv; v_new -> v -> q -> dq; dS -> k;
// T -> dk; Mb -> row partials; dkp stays in registers.
// 16 x 2048 x 16 heads: 220 us with half of the lanes idle in the epilogues, 184 now (HBM: 1.1 GB, 164 us).
constexpr int kChunkSmem = 9 * kTile + 4 * C * 4 + 16 * 4 + 64 + 64;
static_assert(3 * (kChunkSmem + 1024) <= 228 * 1024, "three CTAs per SM");

__global__ void __launch_bounds__(256, 3) gdn_tc_chunk_bwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* XdO = sm;              // swizzled
  uint8_t* Xz = XdO + kTile;      // un-swizzled
  uint8_t* Xe = Xz + kTile;       // -dv_new (un-swizzled), then -e and dv (swizzled)
  uint8_t* Xvn = Xe + kTile;      // v_new (un-swizzled), then v, q, dq (swizzled)
  uint8_t* Xs = Xvn + kTile;      // S0 (un-swizzled)
  uint8_t* Xk = Xs + kTile;       // dS (un-swizzled), then k (swizzled)
  uint8_t* Xt = Xk + kTile;       // T (un-swizzled), then dk (swizzled)
  uint8_t* Xpg = Xt + kTile;      // dP Gamma
  uint8_t* Xy = Xpg + kTile;      // Y, then Mb
  float* gam = reinterpret_cast<float*>(Xy + kTile);
  float* bet = gam + C;
  float* dd = bet + C;
  float* rr = dd + C;
  float* dgo = reinterpret_cast<float*>(Xy);  // [4][C] per-row dgam / dbeta partials of the column quarters, over Mb
  float* dbo = dgo + 4 * C;
  float* red = rr + C;            // [0,8) <dS,S0> per warp, [8,16) sum of k.dkp per warp
  uint64_t* mbar = reinterpret_cast<uint64_t*>(red + 16);  // [0] MMA; loads: [1] first tiles, [2] S0 and dS, [3] k and v, [4] q
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, c = blockIdx.y, b = bh / p.H, h = bh % p.H, t0 = c * C;
  const size_t ci = (size_t)bh * p.n + c;
  const int imax = min(C, p.T - t0);
  auto row = [&](int i) { return ((size_t)(b * p.T + t0 + i) * p.H + h); };
  // this thread's row and 16 columns of every result
  const int i = 32 * (warp & 1) + lane, qd = (warp & 2) + (warp >> 2), j0 = 16 * qd;
  auto block = [&](uint32_t taddr, float (&v)[16]) { ld_acc16(taddr, warp, 16 * (warp >> 2), v); };
  auto row16 = [&](const float* v, float (&e)[16]) {  // per-row scalars of the same 16 columns
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float4 q = *reinterpret_cast<const float4*>(v + j0 + 4 * x);
      e[4 * x] = q.x; e[4 * x + 1] = q.y; e[4 * x + 2] = q.z; e[4 * x + 3] = q.w;
    }
  };

  if (tid == 32) {
    for (int m = 0; m < 5; ++m) tc::mbar_init(mbar + m, 1);
    tc::mbar_fence_init();
    tc::mbar_expect_tx(mbar + 1, 4 * kTile);
    tc::bulk_load(tc::smem_u32(Xe), p.dvn + ci * C * W, kTile, mbar + 1);
    tc::bulk_load(tc::smem_u32(Xt), p.Tm + ci * C * C, kTile, mbar + 1);
    tc::bulk_load(tc::smem_u32(Xvn), p.vn + ci * C * W, kTile, mbar + 1);
    tc::tma_load_4d(tc::smem_u32(XdO), &maps.dO, 0, h, t0, b, mbar + 1);
    tc::mbar_expect_tx(mbar + 2, 2 * kTile);
    tc::bulk_load(tc::smem_u32(Xs), p.hs + ci * W * W, kTile, mbar + 2);
    tc::bulk_load(tc::smem_u32(Xk), p.dhs + ci * W * W, kTile, mbar + 2);
    tc::tma_prefetch_4d(&maps.k, 0, h, t0, b);  // their buffers are still occupied
    tc::tma_prefetch_4d(&maps.v, 0, h, t0, b);
    tc::tma_prefetch_4d(&maps.q, 0, h, t0, b);
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, 128);
    tc::tmem_relinquish();
  }
  if (tid >= 64 && tid < 64 + C) {
    const int x = tid - 64;
    gam[x] = p.gam[ci * C + x];
    bet[x] = x < imax ? p.beta[row(x)] : 0.f;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const float glast = gam[C - 1], L = exp_nonpos(glast);
  if (tid < C) {
    dd[tid] = exp_nonpos(gam[tid]);
    rr[tid] = exp_nonpos(glast - gam[tid]);
  }
  const uint32_t tA = *tslot, tB = tA + 32, tK = tA + 64, tQ = tA + 96;
  uint32_t ph = 0;
  bool ok = (tc::smem_u32(sm) & 1023u) == 0 && tc::mbar_wait(mbar + 1, 0);
  auto wait_mma = [&]() {
    if (ok) ok = tc::mbar_wait(mbar, ph);
    ph ^= 1;
    tc::fence_after_sync();
    ok = __all_sync(0xffffffffu, ok);  // warp-uniform: whole warps read the accumulators
  };
  auto publish = [&]() {  // shared-memory writes -> operands of the next batch
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  };
  // ---- batch 1 ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tA, tc::mnmajor_tile(Xt, C), tc::mnmajor_tile(Xe, W), 64, W, C, false);
    tc::issue_gemm<true>(tB, tc::kmajor_sw128_tile(XdO, kTile), tc::kmajor_tile(Xvn, W), 64, 64, W, false);
    tc::mma_commit(mbar);
  }
  __syncthreads();  // dd, rr visible
  const float gi = gam[i], bi = bet[i], di = dd[i], ri = rr[i];
  wait_mma();
  if (ok) {
    float v[16];
    block(tA, v);  // -e, swizzled like a TMA tile: scaled by -beta in place later, the same bytes leave as dv
#pragma unroll
    for (int x = 0; x < 2; ++x) sts16(Xe, sw_unit(i, (j0 >> 3) + x), pack8(&v[8 * x]));
    block(tB, v);  // dP Gamma, lower triangle incl. diagonal
    float gj[16];
    row16(gam, gj);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const float val = v[q] * exp_nonpos(gi - gj[q]);  // unconditional: the exponentials overlap
      v[q] = (j0 + q <= i) ? val : 0.f;
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) sts16(Xpg, tc::kmajor_unit(i, (j0 >> 3) + x, C), pack8(&v[8 * x]));
    scale_rows(XdO, dd, 256);  // for DQ, at the end
  }
  if (ok) ok = tc::mbar_wait(mbar + 2, 0);  // S0, dS
  publish();
  // ---- batch 2 ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tA, tc::kmajor_sw128_tile(Xe, kTile), tc::kmajor_tile(Xs, W), 64, W, W, false);
    tc::issue_gemm<true>(tB, tc::kmajor_tile(Xvn, W), tc::kmajor_tile(Xk, W), 64, W, W, false);
    tc::issue_gemm<true>(tQ, tc::kmajor_sw128_tile(XdO, kTile), tc::kmajor_tile(Xs, W), 64, W, W, false);
    tc::mma_commit(mbar);
  }
  {  // <dS, S0>
    float part = 0.f;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      float a[8], s[8];
      unpack8(*reinterpret_cast<const uint4*>(Xk + (tid + 256 * x) * 16), a);
      unpack8(*reinterpret_cast<const uint4*>(Xs + (tid + 256 * x) * 16), s);
#pragma unroll
      for (int y = 0; y < 8; ++y) part = fmaf(a[y], s[y], part);
    }
    part = warp_sum(part);
    if (lane == 0) red[warp] = part;
  }
  tc::fence_async_smem();
  __syncthreads();  // every thread is done with dS before the copy engine overwrites the buffer
  wait_mma();
  if (ok && tid == 128) {  // v_new and dS are dead: v and k take their places
    tc::mbar_expect_tx(mbar + 3, 2 * kTile);
    tc::tma_load_4d(tc::smem_u32(Xk), &maps.k, 0, h, t0, b, mbar + 3);
    tc::tma_load_4d(tc::smem_u32(Xvn), &maps.v, 0, h, t0, b, mbar + 3);
  }
  uint4 dkp[2] = {zero16(), zero16()};  // r (v_new dS^T), this lane's 16 columns
  if (ok) {
    float v[16];
    block(tA, v);
#pragma unroll
    for (int x = 0; x < 2; ++x) sts16(Xz, tc::kmajor_unit(i, (j0 >> 3) + x, W), pack8(&v[8 * x]));
    block(tB, v);
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] *= ri;
    dkp[0] = pack8(v);
    dkp[1] = pack8(v + 8);
  }
  if (ok) ok = tc::mbar_wait(mbar + 3, 0);  // k, v
  publish();
  // ---- batch 3 ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tA, tc::kmajor_sw128_tile(Xe, kTile), tc::kmajor_sw128_tile(Xvn, kTile), 64, 64, W, false);
    tc::issue_gemm<true>(tB, tc::kmajor_tile(Xz, W), tc::kmajor_sw128_tile(Xk, kTile), 64, 64, W, false);
    tc::mma_commit(mbar);
    tc::issue_gemm<true>(tK, tc::kmajor_sw128_tile(Xk, kTile), tc::kmajor_sw128_tile(Xk, kTile), 64, 64, W, false);  // for batch 4
  }
  float vdot = 0.f, kz = 0.f;  // e_i . v_i and k_i . z_i: the diagonals of the two products
  wait_mma();
  if (ok) {  // Y[i][m] = beta_m ((e_i . v_m) + d_m (z_i . k_m))
    float ha[16], hb[16];
    block(tA, ha);
    block(tB, hb);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      vdot = (j0 + q == i) ? -ha[q] : vdot;
      kz = (j0 + q == i) ? hb[q] : kz;
    }
    float bj[16], dj[16];
    row16(bet, bj);
    row16(dd, dj);
#pragma unroll
    for (int q = 0; q < 16; ++q) ha[q] = bj[q] * fmaf(dj[q], hb[q], -ha[q]);
#pragma unroll
    for (int x = 0; x < 2; ++x) sts16(Xy, tc::kmajor_unit(i, (j0 >> 3) + x, C), pack8(&ha[8 * x]));
  }
  publish();
  if (ok && tid == 128) {  // q takes the place of v
    tc::mbar_expect_tx(mbar + 4, kTile);
    tc::tma_load_4d(tc::smem_u32(Xvn), &maps.q, 0, h, t0, b, mbar + 4);
  }
  // ---- batch 4 ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tA, tc::kmajor_tile(Xy, C), tc::kmajor_tile(Xt, C), 64, 64, C, false);
    tc::mma_commit(mbar);
  }
  if (ok)  // -e has served as an operand for the last time: dv = beta e in place
    for (int u = tid; u < 512; u += 256) {
      uint4* unit = reinterpret_cast<uint4*>(Xe + 16 * u);
      *unit = tc::scale_bf16x8(*unit, -bet[u >> 3]);
    }
  wait_mma();
  float db_own = 0.f, dg_own = 0.f;
  if (ok) {  // Xy <- Mb = beta_i M, M = -dA Gamma strictly lower, zeros elsewhere
    float ha[16], hk[16], gj[16], rs = 0.f;
    block(tA, ha);
    block(tK, hk);
    row16(gam, gj);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const float mv = -ha[q] * exp_nonpos(gi - gj[q]);
      const float M = (j0 + q < i) ? mv : 0.f;
      rs = fmaf(M, hk[q], rs);
      ha[q] = bi * M;
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) sts16(Xy, tc::kmajor_unit(i, (j0 >> 3) + x, C), pack8(&ha[8 * x]));
    db_own = vdot + di * kz + rs;
    dg_own = 2.f * bi * (di * kz + rs);
  }
  if (ok) ok = tc::mbar_wait(mbar + 4, 0);  // q
  publish();
  // ---- batch 5 ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tA, tc::mnmajor_tile(Xpg, C), tc::mnmajor_sw128_tile(Xvn, kTile), 64, W, C, false);
    tc::issue_gemm<true>(tA, tc::kmajor_tile(Xy, C), tc::mnmajor_sw128_tile(Xk, kTile), 64, W, C, true);
    tc::issue_gemm<true>(tA, tc::mnmajor_tile(Xy, C), tc::mnmajor_sw128_tile(Xk, kTile), 64, W, C, true);
    tc::issue_gemm<true>(tQ, tc::kmajor_tile(Xpg, C), tc::mnmajor_sw128_tile(Xk, kTile), 64, W, C, true);
    tc::mma_commit(mbar);
  }
  wait_mma();
  float rho = 0.f;
  if (ok) {
    float v[16], kd = 0.f, qdot = 0.f;
    block(tA, v);
#pragma unroll
    for (int x = 0; x < 2; ++x) {  // dk = dkp + (dPG^T q + (Mb + Mb^T) k) + beta d z, over T
      const int c8 = (j0 >> 3) + x;
      float e[8], z[8], kr[8];
      unpack8(dkp[x], e);
      unpack8(*reinterpret_cast<const uint4*>(Xz + tc::kmajor_unit(i, c8, W)), z);
      unpack8(*reinterpret_cast<const uint4*>(Xk + sw_unit(i, c8)), kr);
#pragma unroll
      for (int y = 0; y < 8; ++y) {
        rho = fmaf(kr[y], e[y], rho);                        // k_i . dkp_i
        const float val = v[8 * x + y] + e[y] + bi * di * z[y];
        kd = fmaf(kr[y], val, kd);                           // k_i . dk_i
        v[8 * x + y] = val;
      }
      sts16(Xt, sw_unit(i, c8), pack8(&v[8 * x]));
    }
    block(tQ, v);
#pragma unroll
    for (int x = 0; x < 2; ++x) {  // dq, assembled over q (each thread rewrites the units it read)
      const int c8 = (j0 >> 3) + x;
      float qr[8];
      unpack8(*reinterpret_cast<const uint4*>(Xvn + sw_unit(i, c8)), qr);
#pragma unroll
      for (int y = 0; y < 8; ++y) qdot = fmaf(qr[y], v[8 * x + y], qdot);
      sts16(Xvn, sw_unit(i, c8), pack8(&v[8 * x]));
    }
    dg_own += qdot - kd;
  }
  {
    const float tot = warp_sum(rho);
    if (lane == 0) red[8 + warp] = tot;  // summed in a fixed order below
  }
  dgo[qd * C + i] = dg_own;  // (every product that read Mb has completed)
  dbo[qd * C + i] = db_own;
  publish();
  if (ok && p.dq32) {
    const size_t row0 = (size_t)(b * p.T + t0) * p.H + h;
    put_wide_tile(p.dq32, Xvn, row0, p.H, W, imax);
    put_wide_tile(p.dk32, Xt, row0, p.H, W, imax);
    put_wide_tile(p.dv32, Xe, row0, p.H, W, imax);
  } else if (ok && tid == 64) {  // rows past the end of the sequence are clipped
    tc::tma_store_4d(&maps.dq, tc::smem_u32(Xvn), 0, h, t0, b);
    tc::tma_store_4d(&maps.dk, tc::smem_u32(Xt), 0, h, t0, b);
    tc::tma_store_4d(&maps.dv, tc::smem_u32(Xe), 0, h, t0, b);
    tc::bulk_commit();
  }
  if (tid < 32) {  // dg = reverse cumulative sum of dgam within the chunk: one warp, two rows per lane
    float base = 0.f, kp = 0.f;
    for (int wv = 0; wv < 8; ++wv) { base += red[wv]; kp += red[8 + wv]; }
    base = L * base + kp;
    const int ra = C - 1 - 2 * tid, rb = ra - 1;
    float a = (dgo[ra] + dgo[C + ra]) + (dgo[2 * C + ra] + dgo[3 * C + ra]);
    float bq = (dgo[rb] + dgo[C + rb]) + (dgo[2 * C + rb] + dgo[3 * C + rb]);
    warp_rcumsum64(a, bq, tid);
    __syncwarp();
    dgo[ra] = base + a;
    dgo[rb] = base + bq;
  }
  __syncthreads();
  if (!ok && tid == 0) atomicExch(p.status, 4);
  if (ok && tid < imax) {
    p.dbeta[row(tid)] = (dbo[tid] + dbo[C + tid]) + (dbo[2 * C + tid] + dbo[3 * C + tid]);
    float dg = dgo[tid];
    const float gin = p.gate[row(tid)];
    if (p.gate_is_log) {
      if (gin < kLogGateFloor) dg = 0.f;
    } else {
      dg = (gin > kGateFloor) ? dg / gin : 0.f;
    }
    p.dgate[row(tid)] = dg;
  }
  if (tid == 64) tc::bulk_wait_read<0>();  // shared memory must outlive the stores
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tA, 128);
}
}  // namespace g64

// ------------------------------------------------------------------ host
mxb_status tc64_run_fwd(TcP& p, cudaStream_t st) {
  RowMaps maps;
  std::memset(&maps, 0, sizeof maps);
  if (!(make_tma_map_bthd(&maps.k, p.k, p.B, p.T, p.H, g64::W) && make_tma_map_bthd(&maps.q, p.q, p.B, p.T, p.H, g64::W) &&
        make_tma_map_bthd(&maps.v, p.v, p.B, p.T, p.H, g64::W) && make_tma_map_bthd(&maps.o, p.out, p.B, p.T, p.H, g64::W)))
    return MXB_ERR_UNSUPPORTED;
  if (MXB_ALLOW_SMEM(g64::kPrepSmem, g64::gdn_tc_prep_kernel) != MXB_OK ||
      MXB_ALLOW_SMEM(g64::kStateFwdSmem, g64::gdn_tc_state_fwd_kernel) != MXB_OK)
    return MXB_ERR_CUDA;
  MXB_LAUNCH("gdn_tc_prep_kernel", st,
             (launch_kernel(g64::gdn_tc_prep_kernel, dim3(p.n, p.B * p.H), 128, g64::kPrepSmem, st, p, maps)));
  if (const int nv = chain_columns(p, p.save)) return chain_fwd(p, maps, nv, st);
  MXB_LAUNCH("gdn_tc_state_fwd_kernel", st,
             (launch_kernel(g64::gdn_tc_state_fwd_kernel, p.B * p.H, 256, g64::kStateFwdSmem, st, p, maps)));
  return check_launch("gdn_tc64 forward");
}
// After a forward that saved its intermediates: reverse state pass, per-chunk pass.
mxb_status tc64_run_bwd(const TcP& p, cudaStream_t st) {
  RowMaps maps;
  std::memset(&maps, 0, sizeof maps);
  if (!(make_tma_map_bthd(&maps.k, p.k, p.B, p.T, p.H, g64::W) && make_tma_map_bthd(&maps.q, p.q, p.B, p.T, p.H, g64::W) &&
        make_tma_map_bthd(&maps.v, p.v, p.B, p.T, p.H, g64::W) && make_tma_map_bthd(&maps.dO, p.dO, p.B, p.T, p.H, g64::W) &&
        make_tma_map_bthd(&maps.dq, p.dq, p.B, p.T, p.H, g64::W) && make_tma_map_bthd(&maps.dk, p.dk, p.B, p.T, p.H, g64::W) &&
        make_tma_map_bthd(&maps.dv, p.dv, p.B, p.T, p.H, g64::W)))
    return MXB_ERR_UNSUPPORTED;
  if (MXB_ALLOW_SMEM(g64::kStateBwdSmem, g64::gdn_tc_state_bwd_kernel) != MXB_OK ||
      MXB_ALLOW_SMEM(g64::kChunkSmem, g64::gdn_tc_chunk_bwd_kernel) != MXB_OK)
    return MXB_ERR_CUDA;
  if (const int nv = chain_columns(p, true)) {
    const mxb_status s = chain_bwd(p, maps, nv, st);
    if (s != MXB_OK) return s;
  } else {
    MXB_LAUNCH("gdn_tc_state_bwd_kernel", st,
               (launch_kernel(g64::gdn_tc_state_bwd_kernel, p.B * p.H, 256, g64::kStateBwdSmem, st, p, maps)));
  }
  MXB_LAUNCH("gdn_tc_chunk_bwd_kernel", st,
             (launch_kernel(g64::gdn_tc_chunk_bwd_kernel, dim3(p.B * p.H, p.n), 256, g64::kChunkSmem, st, p, maps)));
  return check_launch("gdn_tc64 backward");
}

}  // namespace mxb
