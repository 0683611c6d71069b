// Gated delta rule - tensor-core backward (tcgen05.mma, TMEM accumulators),
// bf16 I/O, fp32 state gradient, chunk 64, Dk = Dv = 128.
//
// Hand-derived backward of the chunked form (the reference differentiates
// gpu/ir.cpp:2352-2550 with MLX autograd; its only VJP, tril(T^T dT T^T,-1) of the
// triangular solve, gpu/gated_delta_cuda_primitive.cpp:104-132, is phase C below).
// With d = E(gam), r = E(gam_last-gam), L = E(gam_last), S0 the state at chunk start
// and dS the state gradient at chunk end:
//
//   gdn_tc_state_bwd_kernel  reverse over chunks, one CTA per (batch, head), operands two chunks ahead:
//       dv_new = P^T dO + r (k dS)
//       dS    <- L dS + (d q)^T dO - w^T dv_new
//   gdn_tc_chunk_bwd_kernel  one CTA per chunk, everything else (the contractions with the saved states S0 and dS
//       included):
//       dq = d (dO S0^T) + (dP*Gamma) k                      dP = tril(dO v_new^T)
//       dw = -dv_new S0^T ; dT = dv_new (v beta)^T + dw (k beta d)^T ; dA = tril(T^T dT T^T,-1)
//       dk = (dP*Gamma)^T q + r (v_new dS^T) + beta d (T^T dw) + (Mb + Mb^T) k,  Mb = -beta dA*Gamma
//       dv = beta (T^T dv_new) ; dbeta, dgam from the same pieces ; dg = reverse cumsum of dgam
//
// A 64 x W bf16 tile stored as 8x8-element blocks ("blocked row-major", umma_tiles.cuh)
// can be read by tcgen05.mma either with the contraction along its columns (K-major) or
// along its rows (MN-major); both views are used on the same staged bytes.
#include <cstring>

#include "gdn_tc.cuh"

namespace mxb {

// One CTA (256 threads) per (batch, head) and NV columns; thread t owns row kk = t & 127 of dS and the
// columns of half t >> 7.  Chunks run in reverse.  The operand tiles are double-buffered (buffer c & 1 for
// chunk c) and requested two chunks ahead, as soon as the products that last read the buffer have completed:
//   group A  k, dO, q rows and the P image   free after k dS
//   group B  the w image                     free after w^T dv_new
// q is scaled in place to diag(E(gam)) q, so that it is contracted with the raw dO tile:
//   dv_new = diag(r) k dS + P^T dO,   dS <- E(gam_last) dS + (d q)^T dO - w^T dv_new.
//
// Bound by the chain dS -> k dS -> dv_new -> w^T dv_new -> dS where the heads are few, by HBM where they fill the GPU.
// P^T dO and (d q)^T dO need no dS: those of chunk c-1 are issued behind w^T dv_new of chunk c and run while dS is
// updated, and q is scaled in the shadow of the k dS before (16 heads of 128, NV = 64: 2.6 -> 1.7 us a chunk).
// (An issuing warp of its own, as in the forward pass, was slower here: 1.8 -> 2.1 us.)
//
// TMA = true: the k, dO and q rows arrive as tensor-map boxes (128-byte swizzle, two 8 KB slabs of 64 columns per
// tile) issued by one thread on the barrier of group A; TMA = false: by cp.async into the same swizzled positions
// (twelve copies per thread and chunk).  The w image is stored in the same swizzled layout by the prep kernel.
// NV: columns of dS per CTA, as in the forward pass.
template <int NV>
constexpr int kStateBwdSmem =
    2 * 16384 + 256 * NV + 2 * 8192 + 2 * 128 * NV + 2 * 16384 + 2 * 16384 + 128 * NV + 3 * C * 4 + 128 + 1024;

template <bool TMA, int NV>
__global__ void __launch_bounds__(256) gdn_tc_state_bwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  static_assert(NV == KD || TMA, "the per-thread staging moves whole rows");
  constexpr int NC = NV / 2;                   // columns per thread
  const int col0 = blockIdx.y * NV;
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Ak = sm;                  // x2 [64 i][128 kk]   k  (swizzled slabs)
  uint8_t* dSop = Ak + 2 * 16384;    // [128 kk][NV j]      bf16 copy of dS
  uint8_t* Pt = dSop + 256 * NV;        // x2 [64 m][64 i]     P   (A = P^T: contraction over rows)
  uint8_t* dOop = Pt + 2 * 8192;     // x2 [64 m][NV j]     dO (swizzled slabs)
  uint8_t* Aq = dOop + 2 * 128 * NV;    // x2 [64 i][128 kk]   q, then diag(E(gam)) q (swizzled slabs)   (A = q^T)
  uint8_t* Aw = Aq + 2 * 16384;      // x2 [64 i][128 kk]   w image (swizzled slabs)                  (A = w^T)
  uint8_t* Bd = Aw + 2 * 16384;      // [64 i][NV j]        -dv_new
  float* rr = reinterpret_cast<float*>(Bd + 128 * NV);
  float* ddn = rr + C;               // x2 E(gam) of the chunk whose q is scaled next (buffer = chunk & 1)
  // [0] MMA completion; per buffer: [1 + buf] group A landed, [3 + buf] w image landed
  uint64_t* mbar = reinterpret_cast<uint64_t*>(ddn + 2 * C);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 8);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kk = tid & 127, half = tid >> 7, j0 = NC * half;
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  const uint32_t sAk = tc::smem_u32(Ak), sPt = tc::smem_u32(Pt), sdO = tc::smem_u32(dOop), sAq = tc::smem_u32(Aq);
  const uint32_t sAw = tc::smem_u32(Aw);

  auto grow = [&](int c, int i) { return ((size_t)(b * p.T + c * C + i) * p.H + h); };
  auto issue_A = [&](int c) {
    if (c >= 0) {
      const size_t ci = (size_t)bh * p.n + c;
      const uint32_t o16 = (c & 1) * 16384;
      if (!TMA) {
        const int imax = min(C, p.T - c * C);
        for (int u = tid; u < 64 * 16; u += 256) {
          const int i = urow16(u), c8 = ucol16(u);
          const bool v = i < imax;
          const size_t g = v ? grow(c, i) * KD + c8 * 8 : 0;
          const uint32_t off = o16 + tc::sw128_unit(i, c8);
          tc::cp_async16(sAk + off, p.k + g, v);
          tc::cp_async16(sdO + off, p.dO + g, v);
          tc::cp_async16(sAq + off, p.q + g, v);
        }
      }
      if (tid == 32) {  // P is a byte image of its operand tile: one bulk copy, completing on the group's barrier
        uint64_t* mb = &mbar[1 + (c & 1)];
        tc::mbar_expect_tx(mb, TMA ? 8192 + 2 * 16384 + 128 * NV : 8192);
        tc::bulk_load(sPt + (c & 1) * 8192, p.P + ci * C * C, 8192, mb);
        if (TMA) {
          for (int sl = 0; sl < 2; ++sl) {
            tc::tma_load_4d(sAk + o16 + sl * 8192, &maps.k, 64 * sl, h, c * C, b, mb);
            if (sl < NV / 64) tc::tma_load_4d(sdO + (c & 1) * 128 * NV + sl * 8192, &maps.dO, col0 + 64 * sl, h, c * C, b, mb);
            tc::tma_load_4d(sAq + o16 + sl * 8192, &maps.q, 64 * sl, h, c * C, b, mb);
          }
        }
      }
    }
    if (!TMA) tc::cp_async_commit();
  };
  auto issue_B = [&](int c) {
    if (c >= 0 && tid == 32) {
      const size_t ci = (size_t)bh * p.n + c;
      tc::mbar_expect_tx(&mbar[3 + (c & 1)], 16384);
      tc::bulk_load(sAw + (c & 1) * 16384, p.w + ci * C * KD, 16384, &mbar[3 + (c & 1)]);
    }
    if (!TMA) tc::cp_async_commit();  // (empty: keeps the group count of the schedule)
  };
  // q of chunk c <- diag(E(gam)) q in place; every thread scales the 16-byte units it would copy itself
  auto scale_q = [&](int c) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int u = tid + 256 * m, i = urow16(u);
      uint4* unit = reinterpret_cast<uint4*>(Aq + (c & 1) * 16384 + tc::sw128_unit(i, ucol16(u)));
      *unit = tc::scale_bf16x8(*unit, ddn[(c & 1) * C + i]);
    }
  };

  if (warp == 0) {
    tc::tmem_alloc(tslot, 512);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int m = 0; m < 5; ++m) tc::mbar_init(&mbar[m], 1);
    tc::mbar_fence_init();
  }
  __syncthreads();  // barriers initialised before the copies can complete on them
  for (int c = p.n - 1; c > p.n - 3; --c) {
    issue_A(c);
    issue_B(c);
  }
  float dS[NC];  // row kk of dS, columns col0 + j0 ..
  if (p.dhT_in) {
    const float4* src = reinterpret_cast<const float4*>(p.dhT_in + ((size_t)bh * p.Dk + kk) * p.Dv + col0 + j0);
#pragma unroll
    for (int x = 0; x < NC / 4; ++x) {
      const float4 t4 = (kk < p.Dk && col0 + j0 + 4 * x < p.Dv) ? __ldg(src + x) : make_float4(0.f, 0.f, 0.f, 0.f);
      dS[4 * x] = t4.x; dS[4 * x + 1] = t4.y; dS[4 * x + 2] = t4.z; dS[4 * x + 3] = t4.w;
    }
  } else {
#pragma unroll
    for (int x = 0; x < NC; ++x) dS[x] = 0.f;
  }
  // Decay factors: rr of the chunk ahead and ddn of the one after it, computed in the shadow of w^T dv_new.
  const size_t gbase = (size_t)bh * p.n * C;
  auto gam_at = [&](int c) { return c >= 0 ? p.gam[gbase + (size_t)c * C + (tid & 63)] : 0.f; };
  auto gam_end = [&](int c) { return c >= 0 ? p.gam[gbase + (size_t)c * C + C - 1] : 0.f; };
  float gl_cur = gam_end(p.n - 1), g_nxt = gam_at(p.n - 2), gl_nxt = gam_end(p.n - 2);
  if (tid < C) {
    const float g = gam_at(p.n - 1);
    rr[tid] = exp_nonpos(gl_cur - g);
    ddn[((p.n - 1) & 1) * C + tid] = exp_nonpos(g);
    ddn[(p.n & 1) * C + tid] = exp_nonpos(g_nxt);
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  uint32_t ph = 0;
  bool ok = true;
  // P^T dO and (d q)^T dO of chunk c (accumulators at 128 and at 256 or 384)
  auto issue_dO = [&](int c) {
    const tc::Tile dO = tc::mnmajor_sw128_tile(dOop + (c & 1) * 128 * NV, 8192);
    tc::issue_gemm<true>(taddr + 128, tc::mnmajor_tile(Pt + (c & 1) * 8192, C), dO, 64, NV, C, false);
    tc::issue_gemm(taddr + 256 + 128 * (c & 1), tc::mnmajor_sw128_tile(Aq + (c & 1) * 16384, 8192), dO, 128, NV, C, false);
  };
  {  // the last chunk's q is scaled here; every later one a chunk ahead
    const int c = p.n - 1;
    if (!TMA) tc::cp_async_wait<2>();
    ok = tc::mbar_wait(&mbar[1 + (c & 1)], 0);
    scale_q(c);
  }

  for (int c = p.n - 1; c >= 0; --c) {
    const size_t ci = (size_t)bh * p.n + c;
    const int buf = c & 1;
    const uint32_t lph = ((p.n - 1 - c) >> 1) & 1;  // phase of this buffer's barriers
    const float L = exp_nonpos(gl_cur);
    const float g_far = gam_at(c - 2), gl_far = gam_end(c - 2);
#pragma unroll
    for (int c8 = 0; c8 < NC / 8; ++c8) {  // dS at chunk end: MMA operand + saved for the chunk kernel
      const uint4 val = make_uint4(tc::pack_bf16(dS[8 * c8], dS[8 * c8 + 1]), tc::pack_bf16(dS[8 * c8 + 2], dS[8 * c8 + 3]),
                                   tc::pack_bf16(dS[8 * c8 + 4], dS[8 * c8 + 5]), tc::pack_bf16(dS[8 * c8 + 6], dS[8 * c8 + 7]));
      sts16(dSop, tc::colblk_unit(kk, NC / 8 * half + c8, KD), val);
    }
    if (tid == 0) tc::bulk_wait_read<0>();  // the previous chunk's -dv_new image has left its tile
    tc::fence_async_smem();
    tc::fence_before_sync();
    ok = __syncthreads_and(ok);  // the barrier also makes the verdict of the bounded waits uniform, so that all
    if (!ok) break;              // threads leave the loop together
    tc::fence_after_sync();
    if (tid == 0) {
      if (c == p.n - 1) issue_dO(c);
      tc::issue_gemm<true>(taddr, tc::kmajor_sw128_tile(Ak + buf * 16384, 8192), tc::colblk_mnmajor_tile(dSop, KD), 64, NV, KD, false);  // k dS
      tc::mma_commit(mbar);
      // dS at chunk end, as the operand-tile image
      tc::bulk_store(p.dhs + ci * KD * KD + KD * col0, tc::smem_u32(dSop), 256 * NV);
      tc::bulk_commit();
    }
    if (c > 0) {  // in the shadow of that product: the next chunk's q (its group was requested a chunk ago)
      if (!TMA) tc::cp_async_wait<1>();
      ok = tc::mbar_wait(&mbar[1 + (buf ^ 1)], ((p.n - c) >> 1) & 1);
      scale_q(c - 1);
    }
    if (ok) ok = tc::mbar_wait(&mbar[3 + buf], lph);  // w image of this chunk
    if (ok) ok = tc::mbar_wait(mbar, ph);
    ph ^= 1;
    tc::fence_after_sync();
    issue_A(c - 2);
    if (ok) {
      // weight-stationary: this thread's row and quarter of the columns (the second half of them in lanes 64-127)
      constexpr int NQ = NV / 4;
      const int i = 32 * (warp & 1) + lane, tc0 = NQ * (warp >> 2), c8 = NV / 16 * ((warp >> 1) & 1) + NQ / 8 * (warp >> 2);
      const float ri = rr[i];
      float fa[NQ], fb[NQ];
      ld_accN(taddr + tc0, warp, fa);
      ld_accN(taddr + 128 + tc0, warp, fb);
#pragma unroll
      for (int x = 0; x < NQ / 8; ++x) {
        float e[8];
#pragma unroll
        for (int y = 0; y < 8; ++y) e[y] = -fmaf(ri, fa[8 * x + y], fb[8 * x + y]);
        sts16(Bd, tc::colblk_unit(i, c8 + x, C), make_uint4(tc::pack_bf16(e[0], e[1]), tc::pack_bf16(e[2], e[3]),
                                                            tc::pack_bf16(e[4], e[5]), tc::pack_bf16(e[6], e[7])));
      }
    }
    if (tid == 0) tc::bulk_wait_read<0>();  // the dS image has left its tile
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (ok && tid == 0) {  // ... - w^T dv_new
      tc::issue_gemm(taddr + 256 + 128 * buf, tc::mnmajor_sw128_tile(Aw + buf * 16384, 8192), tc::colblk_mnmajor_tile(Bd, C), 128, NV, C,
                     true);
      tc::mma_commit(mbar);
      if (c > 0) issue_dO(c - 1);  // (completes with the next commit)
      // -dv_new as the operand-tile image
      tc::bulk_store(p.dvn + ci * C * KD + C * col0, tc::smem_u32(Bd), 128 * NV);
      tc::bulk_commit();
    }
    if (tid < C && c > 0) {
      rr[tid] = exp_nonpos(gl_nxt - g_nxt);
      ddn[buf * C + tid] = exp_nonpos(g_far);
    }
    gl_cur = gl_nxt; g_nxt = g_far; gl_nxt = gl_far;
    if (ok) {
      ok = tc::mbar_wait(mbar, ph);
      ph ^= 1;
    }
    tc::fence_after_sync();
    issue_B(c - 2);
    if (ok) {
      float a[NC];
      ld_accN(taddr + 256 + 128 * buf + j0, warp, a);
#pragma unroll
      for (int jj = 0; jj < NC; ++jj) dS[jj] = fmaf(L, dS[jj], a[jj]);
    }
    tc::fence_before_sync();
  }
  if (!TMA) tc::cp_async_wait<0>();
  if (tid == 0) tc::bulk_wait_read<0>();  // shared memory must outlive the copies
  if (!ok && tid == 0) atomicExch(p.status, 3);
  if (ok && p.dh0 && kk < p.Dk) {
    float4* dst = reinterpret_cast<float4*>(p.dh0 + ((size_t)bh * p.Dk + kk) * p.Dv + col0 + j0);
#pragma unroll
    for (int x = 0; x < NC / 4; ++x)
      if (col0 + j0 + 4 * x < p.Dv) dst[x] = make_float4(dS[4 * x], dS[4 * x + 1], dS[4 * x + 2], dS[4 * x + 3]);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 512);
}

// ------------------------------------------------- chunk backward
// One CTA per chunk does everything that is not the sequential state pass.  With e = T^T dv_new, z = T^T dw = -e S0^T
// (dw = -dv_new S0^T never needs to be formed), Gamma_ij = E(gam_i - gam_j):
//   batch 1   -e = T^T (-dv_new)                    dP = dO v_new^T                -> dPG = dP*Gamma (lower incl. diagonal)
//   batch 2   DQ = (d dO) S0^T   (stays in TMEM)    z = (-e) S0^T                  (dO is scaled by d in place first)
//   batch 3   r (v_new dS^T) -> dkp                                                 <dS, S0> on the side
//   batch 4   (-e) v^T, z k^T   -> Y = T^T dT = beta_m (e.v_m + d_m z.k_m)
//   batch 5   dA = tril(Y T^T, -1), k k^T           -> M = -dA*Gamma, Mb = beta_i M
//   batch 6   DQ += dPG k                            dPG^T q + Mb k + Mb^T k
//   dq = DQ      dk = dkp + batch 6 + beta d z      dv = beta e      dbeta = e.v + d (k.z) + sum_j M_ij (k_i.k_j)
//   dgam_i = q_i.dq_i - k_i.dk_i + 2 beta_i (d_i (k_i.z_i) + sum_j M_ij (k_i.k_j)),  dgam_last += L <dS,S0> + sum_i k_i.dkp_i
// (the row and column sums over Gamma of the P and A terms are exactly the parts of q.dq and k.dk that come from
// dPG and Mb, so they need no products of their own).
//
// 256 TMEM columns and 107 KB of shared memory: two CTAs share an SM.  Every buffer is reused as soon as it is dead:
//   XdO   dO (TMA tile) -> d dO -> z                      Xe   -dv_new image -> -e -> dv = beta e on its way out
//   Xvn   v_new image -> v (TMA) -> q (TMA) -> dq         R1   S0 image -> dS image -> k (TMA) | dkp -> dk
// TMEM: [0,64) -e, then DQ until the end; [64,128) the other products one after the other, [128,160) k k^T.  Every
// product is issued in the weight-stationary form, whose M = 64 accumulators fill all 128 lanes: each thread has a row
// (i) and a quarter of the columns (16 of 64, 32 of 128) in every epilogue.
// Bound by the six batches that follow one another within a CTA (HBM: 1.77 GB, 0.27 ms at 8 x 4096 x 16 heads): with
// half of the lanes idle in every epilogue 404 us, this 365 us.  Grid = (batch*head, chunk) with batch*head fastest: neighbouring CTAs read
// neighbouring heads of the same time steps (one contiguous row of the token tensors between them), and the chunks
// the reverse state pass wrote last are read first.
constexpr int kChunkBwdSmem = 3 * 16384 + 32768 + 3 * 8192 + 12 * C * 4 + 16 * 4 + 64 + 64 + 1024;

__global__ void __launch_bounds__(256, 2) gdn_tc_chunk_bwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* XdO = sm;                // [64][128] dO (swizzled TMA tile), d dO in place, then z (blocked layout)
  uint8_t* Xe = XdO + 16384;        // [64][128] -dv_new image (blocked), then -e and finally dv (swizzled like a TMA tile)
  uint8_t* Xvn = Xe + 16384;        // [64][128] v_new image, then v, then q (swizzled TMA tiles), then dq in place
  uint8_t* R1 = Xvn + 16384;        // [128][128] S0 image, then dS image, then k (swizzled TMA tile) | dkp -> dk (swizzled)
  uint8_t* Xk = R1;
  uint8_t* Xdk = R1 + 16384;
  uint8_t* Xt = R1 + 32768;         // [64][64]  T
  uint8_t* Xpg = Xt + 8192;         // [64][64]  dP*Gamma
  uint8_t* Xy = Xpg + 8192;         // [64][64]  Y, then Mb
  float* gam = reinterpret_cast<float*>(Xy + 8192);
  float* bet = gam + C;
  float* dd = bet + C;
  float* rr = dd + C;
  float* dgo = rr + C;              // [4][C] per-row dgam / dbeta partials of the column quarters
  float* dbo = dgo + 4 * C;
  float* red = dbo + 4 * C;         // [0,8) <dS,S0> per warp, [8,16) sum of k.dkp per warp
  // [0] MMA, [6] second MMA barrier of the last batch; loads: [1] -dv_new/T/dO/v_new, [2] S0, [3] dS, [4] k/v, [5] q
  uint64_t* mbar = reinterpret_cast<uint64_t*>(red + 16);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 8);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, c = blockIdx.y, b = bh / p.H, h = bh % p.H, t0 = c * C;
  const size_t ci = (size_t)bh * p.n + c;
  const int imax = min(C, p.T - t0);
  auto row = [&](int i) { return ((size_t)(b * p.T + t0 + i) * p.H + h); };
  // this thread's row and column quarter of every result; tc16 / tc32: its TMEM columns of a [64][64] / [64][128] result
  const int i = 32 * (warp & 1) + lane, qd = (warp & 2) + (warp >> 2), n16 = 16 * qd;
  const int tc16 = 16 * (warp >> 2), tc32 = 32 * (warp >> 2);
  // sixteen per-row scalars of this thread's columns of a [64][64] result
  auto row16 = [&](const float* v, float (&e)[16]) {
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float4 q = *reinterpret_cast<const float4*>(v + n16 + 4 * x);
      e[4 * x] = q.x; e[4 * x + 1] = q.y; e[4 * x + 2] = q.z; e[4 * x + 3] = q.w;
    }
  };

  // prologue latencies side by side: warp 0 allocates TMEM, one thread of warp 1 initialises the barriers and issues
  // the first copies, warps 2-3 fetch the per-row scalars
  if (tid == 32) {
    for (int m = 0; m < 7; ++m) tc::mbar_init(mbar + m, 1);
    tc::mbar_fence_init();
    tc::mbar_expect_tx(mbar + 1, 3 * 16384 + 8192);
    tc::bulk_load(tc::smem_u32(Xe), p.dvn + ci * C * KD, 16384, mbar + 1);  // byte images of the operand tiles
    tc::bulk_load(tc::smem_u32(Xt), p.Tm + ci * C * C, 8192, mbar + 1);
    tc::bulk_load(tc::smem_u32(Xvn), p.vn + ci * C * KD, 16384, mbar + 1);
    for (int sl = 0; sl < 2; ++sl) tc::tma_load_4d(tc::smem_u32(XdO) + 8192 * sl, &maps.dO, 64 * sl, h, t0, b, mbar + 1);
    tc::mbar_expect_tx(mbar + 2, 32768);
    tc::bulk_load(tc::smem_u32(R1), p.hs + ci * KD * KD, 32768, mbar + 2);
    // the operands whose buffers are still occupied are pulled into L2 now, so that their copies find them on chip
    tc::bulk_prefetch_l2(p.dhs + ci * KD * KD, 32768);
    for (int sl = 0; sl < 2; ++sl) {
      tc::tma_prefetch_4d(&maps.k, 64 * sl, h, t0, b);
      tc::tma_prefetch_4d(&maps.v, 64 * sl, h, t0, b);
      tc::tma_prefetch_4d(&maps.q, 64 * sl, h, t0, b);
    }
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, 256);
    tc::tmem_relinquish();
  }
  if (tid >= 64 && tid < 64 + C) {
    const int r = tid - 64;
    gam[r] = p.gam[ci * C + r];
    bet[r] = r < imax ? p.beta[row(r)] : 0.f;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const float glast = gam[C - 1], L = exp_nonpos(glast);
  if (tid < C) {
    dd[tid] = exp_nonpos(gam[tid]);
    rr[tid] = exp_nonpos(glast - gam[tid]);
  }
  const uint32_t tA = *tslot, tB = tA + 64, tK = tA + 128;
  bool ok = tc::mbar_wait(mbar + 1, 0);
  uint32_t ph = 0;
  // ---- batch 1: -e = T^T (-dv_new) (both operands contracted over their rows), dP = dO v_new^T ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tA, tc::mnmajor_tile(Xt, C), tc::colblk_mnmajor_tile(Xe, C), 64, 128, C, false);
    tc::issue_gemm<true>(tB, tc::kmajor_sw128_tile(XdO, 8192), tc::colblk_kmajor_tile(Xvn, C), 64, 64, KD, false);
    tc::mma_commit(mbar);
  }
  __syncthreads();  // dd, rr visible
  const float gi = gam[i], bi = bet[i], di = dd[i], ri = rr[i];
  const float bd_i = bi * di;
  if (ok) ok = tc::mbar_wait(mbar, ph);
  ph ^= 1;
  tc::fence_after_sync();
  ok = __all_sync(0xffffffffu, ok);  // warp-uniform: the epilogues below shuffle with a full mask
  if (ok) {
    // -e goes back over the operand it was computed from (its MMA is complete), in the swizzled layout of a TMA
    // tile: scaled by -beta in place later, the same bytes leave as dv through a tiled store
    {
      float f[32];
      ld_acc32(tA, warp, tc32, f);
#pragma unroll
      for (int x = 0; x < 4; ++x) sts16(Xe, tc::sw128_unit(i, 4 * qd + x), pack8(&f[8 * x]));
    }
    {  // dP * Gamma, lower triangle incl. diagonal
      float hq[16], gj[16];
      ld_acc16(tB, warp, tc16, hq);
      row16(gam, gj);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const float val = hq[q] * exp_nonpos(gi - gj[q]);  // unconditional: the exponentials overlap
        hq[q] = (n16 + q <= i) ? val : 0.f;
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) sts16(Xpg, tc::kmajor_unit(i, 2 * qd + x, C), pack8(&hq[8 * x]));
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {  // dO <- diag(d) dO in place, so that DQ can take dPG k on top later
      const int u = tid + 256 * m, r = urow16(u);
      uint4* unit = reinterpret_cast<uint4*>(XdO + tc::sw128_unit(r, ucol16(u)));
      *unit = tc::scale_bf16x8(*unit, dd[r]);
    }
  }
  if (ok) ok = tc::mbar_wait(mbar + 2, 0);  // S0
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // ---- batch 2: DQ = (d dO) S0^T, z = (-e) S0^T ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tA, tc::kmajor_sw128_tile(XdO, 8192), tc::colblk_kmajor_tile(R1, KD), 64, 128, KD, false);
    tc::issue_gemm<true>(tB, tc::kmajor_sw128_tile(Xe, 8192), tc::colblk_kmajor_tile(R1, KD), 64, 128, KD, false);
    tc::mma_commit(mbar);  // one commit: z overwrites d dO and dS overwrites S0, which DQ reads as well
  }
  uint4 s0u[8];  // this thread's 8 units of S0, kept for <dS, S0> (the buffer is about to be reused)
#pragma unroll
  for (int x = 0; x < 8; ++x) s0u[x] = *reinterpret_cast<const uint4*>(R1 + (tid + 256 * x) * 16);
  tc::fence_async_smem();
  __syncthreads();  // every thread has taken its units of S0 before the copy engine overwrites the buffer
  if (ok) ok = tc::mbar_wait(mbar, ph);
  ph ^= 1;
  tc::fence_after_sync();
  ok = __all_sync(0xffffffffu, ok);  // warp-uniform: the epilogues below shuffle with a full mask
  if (ok && tid == 0) {  // S0 is dead in shared memory: dS comes into the same buffer behind the epilogue
    tc::mbar_expect_tx(mbar + 3, 32768);
    tc::bulk_load(tc::smem_u32(R1), p.dhs + ci * KD * KD, 32768, mbar + 3);
  }
  if (ok) {  // z -> bf16 operand over the dead dO tile (blocked layout)
    float f[32];
    ld_acc32(tB, warp, tc32, f);
#pragma unroll
    for (int x = 0; x < 4; ++x) sts16(XdO, tc::kmajor_unit(i, 4 * qd + x, KD), pack8(&f[8 * x]));
  }
  if (ok) ok = tc::mbar_wait(mbar + 3, 0);  // dS
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // ---- batch 3: v_new dS^T ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tB, tc::colblk_kmajor_tile(Xvn, C), tc::colblk_kmajor_tile(R1, KD), 64, 128, KD, false);
    tc::mma_commit(mbar);
  }
  {  // <dS, S0>
    float part = 0.f;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      float a[8], bq[8];
      unpack8(*reinterpret_cast<const uint4*>(R1 + (tid + 256 * x) * 16), a);
      unpack8(s0u[x], bq);
#pragma unroll
      for (int y = 0; y < 8; ++y) part = fmaf(a[y], bq[y], part);
    }
    part = warp_sum(part);
    if (lane == 0) red[warp] = part;
  }
  tc::fence_async_smem();
  __syncthreads();  // every thread is done with dS before the copy engine overwrites the buffer
  if (ok) ok = tc::mbar_wait(mbar, ph);
  ph ^= 1;
  tc::fence_after_sync();
  ok = __all_sync(0xffffffffu, ok);  // warp-uniform: the epilogues below shuffle with a full mask
  if (ok && tid == 128) {  // v_new and dS are dead: k and v take their places
    tc::mbar_expect_tx(mbar + 4, 2 * 16384);
    for (int sl = 0; sl < 2; ++sl) {
      tc::tma_load_4d(tc::smem_u32(Xk) + 8192 * sl, &maps.k, 64 * sl, h, t0, b, mbar + 4);
      tc::tma_load_4d(tc::smem_u32(Xvn) + 8192 * sl, &maps.v, 64 * sl, h, t0, b, mbar + 4);
    }
  }
  if (ok) {  // dkp = r (v_new dS^T), kept as bf16 where dk will be assembled
    float f[32];
    ld_acc32(tB, warp, tc32, f);
#pragma unroll
    for (int jj = 0; jj < 32; ++jj) f[jj] *= ri;
#pragma unroll
    for (int x = 0; x < 4; ++x) sts16(Xdk, tc::sw128_unit(i, 4 * qd + x), pack8(&f[8 * x]));
  }
  if (ok) ok = tc::mbar_wait(mbar + 4, 0);  // k, v
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // ---- batch 4: (-e) v^T and z k^T; their column-scaled sum is Y = T^T dT (dT is never formed) ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tB, tc::kmajor_sw128_tile(Xe, 8192), tc::kmajor_sw128_tile(Xvn, 8192), 64, 64, KD, false);
    tc::issue_gemm<true>(tB + 32, tc::kmajor_tile(XdO, KD), tc::kmajor_sw128_tile(Xk, 8192), 64, 64, KD, false);
    tc::mma_commit(mbar);
    tc::issue_gemm<true>(tK, tc::kmajor_sw128_tile(Xk, 8192), tc::kmajor_sw128_tile(Xk, 8192), 64, 64, KD, false);  // k k^T, for batch 5
  }
  float vdot = 0.f, kz = 0.f;  // e_i . v_i and k_i . z_i: the diagonals of the two products of this batch
  if (ok) ok = tc::mbar_wait(mbar, ph);
  ph ^= 1;
  tc::fence_after_sync();
  ok = __all_sync(0xffffffffu, ok);  // warp-uniform: the epilogues below shuffle with a full mask
  if (ok) {  // Y[i][m] = beta_m ((e_i . v_m) + d_m (z_i . k_m))
    float ha[16], hb[16], dj[16], bj[16];
    ld_acc16(tB, warp, tc16, ha);
    ld_acc16(tB + 32, warp, tc16, hb);
    row16(dd, dj);
    row16(bet, bj);
#pragma unroll
    for (int q = 0; q < 16; ++q) {  // the thread whose columns contain column i picks the two row dots off the diagonal
      vdot = (n16 + q == i) ? -ha[q] : vdot;
      kz = (n16 + q == i) ? hb[q] : kz;
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) ha[q] = bj[q] * fmaf(dj[q], hb[q], -ha[q]);
#pragma unroll
    for (int x = 0; x < 2; ++x) sts16(Xy, tc::kmajor_unit(i, 2 * qd + x, C), pack8(&ha[8 * x]));
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();  // also: every thread is done with v
  tc::fence_after_sync();
  if (ok && tid == 128) {  // q takes the place of v
    tc::mbar_expect_tx(mbar + 5, 16384);
    for (int sl = 0; sl < 2; ++sl) tc::tma_load_4d(tc::smem_u32(Xvn) + 8192 * sl, &maps.q, 64 * sl, h, t0, b, mbar + 5);
  }
  // ---- batch 5: dA = tril(Y T^T, -1) ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tB, tc::kmajor_tile(Xy, C), tc::kmajor_tile(Xt, C), 64, 64, C, false);
    tc::mma_commit(mbar);
  }
  if (ok) {  // -e has served as an operand and in the row dots for the last time (barrier above): dv = beta e in place
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int u = tid + 256 * m, r = urow16(u);
      uint4* unit = reinterpret_cast<uint4*>(Xe + tc::sw128_unit(r, ucol16(u)));
      *unit = tc::scale_bf16x8(*unit, -bet[r]);
    }
  }
  if (ok) ok = tc::mbar_wait(mbar, ph);
  ph ^= 1;
  tc::fence_after_sync();
  ok = __all_sync(0xffffffffu, ok);  // warp-uniform: the epilogues below shuffle with a full mask
  float db_own = 0.f, dg_own = 0.f;
  if (ok) {  // Xy <- Mb = beta_i M, M = -dA*Gamma strictly lower, zeros elsewhere
    float ha[16], hk[16], gj[16];
    ld_acc16(tB, warp, tc16, ha);
    ld_acc16(tK, warp, tc16, hk);
    row16(gam, gj);
    float rs = 0.f;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const float mv = -ha[q] * exp_nonpos(gi - gj[q]);  // unconditional: the exponentials overlap
      const float M = (n16 + q < i) ? mv : 0.f;
      rs = fmaf(M, hk[q], rs);
      ha[q] = bi * M;
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) sts16(Xy, tc::kmajor_unit(i, 2 * qd + x, C), pack8(&ha[8 * x]));
    db_own = vdot + di * kz + rs;
    dg_own = 2.f * bi * (di * kz + rs);
  }
  if (ok) ok = tc::mbar_wait(mbar + 5, 0);  // q
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // ---- batch 6: dPG^T q + Mb k + Mb^T k (one tile read K-major and MN-major), committed first: the dk epilogue
  //      runs while DQ += dPG k is still on the tensor core ----
  if (ok && tid == 0) {
    tc::issue_gemm<true>(tB, tc::mnmajor_tile(Xpg, C), tc::mnmajor_sw128_tile(Xvn, 8192), 64, 128, C, false);
    tc::issue_gemm<true>(tB, tc::kmajor_tile(Xy, C), tc::mnmajor_sw128_tile(Xk, 8192), 64, 128, C, true);
    tc::issue_gemm<true>(tB, tc::mnmajor_tile(Xy, C), tc::mnmajor_sw128_tile(Xk, 8192), 64, 128, C, true);
    tc::mma_commit(mbar + 6);
    tc::issue_gemm<true>(tA, tc::kmajor_tile(Xpg, C), tc::mnmajor_sw128_tile(Xk, 8192), 64, 128, C, true);
    tc::mma_commit(mbar);
  }
  if (ok) ok = tc::mbar_wait(mbar + 6, 0);
  tc::fence_after_sync();
  ok = __all_sync(0xffffffffu, ok);  // warp-uniform: the epilogues below shuffle with a full mask
  float rho = 0.f;
  if (ok) {  // dk = dkp + (dPG^T q + (Mb + Mb^T) k) + beta d z, assembled over dkp (each thread rewrites the units it read)
    float f[32], r4[4] = {0.f, 0.f, 0.f, 0.f}, k4[4] = {0.f, 0.f, 0.f, 0.f};
    ld_acc32(tB, warp, tc32, f);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int c8 = 4 * qd + x;
      float e[8], z[8], kr[8];
      unpack8(*reinterpret_cast<const uint4*>(Xdk + tc::sw128_unit(i, c8)), e);
      unpack8(*reinterpret_cast<const uint4*>(XdO + tc::kmajor_unit(i, c8, KD)), z);
      unpack8(*reinterpret_cast<const uint4*>(Xk + tc::sw128_unit(i, c8)), kr);
#pragma unroll
      for (int y = 0; y < 8; ++y) {
        r4[x] = fmaf(kr[y], e[y], r4[x]);              // k_i . dkp_i
        const float val = f[8 * x + y] + e[y] + bd_i * z[y];
        k4[x] = fmaf(kr[y], val, k4[x]);               // k_i . dk_i
        f[8 * x + y] = val;
      }
      sts16(Xdk, tc::sw128_unit(i, c8), pack8(&f[8 * x]));
    }
    rho = (r4[0] + r4[1]) + (r4[2] + r4[3]);
    dg_own -= (k4[0] + k4[1]) + (k4[2] + k4[3]);
  }
  if (ok) ok = tc::mbar_wait(mbar, ph);  // every product has completed
  ph ^= 1;
  tc::fence_after_sync();
  ok = __all_sync(0xffffffffu, ok);  // warp-uniform: the epilogues below shuffle with a full mask
  if (ok) {  // dq, assembled over q (each thread rewrites the units it read)
    float f[32], q4[4] = {0.f, 0.f, 0.f, 0.f};
    ld_acc32(tA, warp, tc32, f);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int c8 = 4 * qd + x;
      float qr[8];
      unpack8(*reinterpret_cast<const uint4*>(Xvn + tc::sw128_unit(i, c8)), qr);
#pragma unroll
      for (int y = 0; y < 8; ++y) q4[x] = fmaf(qr[y], f[8 * x + y], q4[x]);
      sts16(Xvn, tc::sw128_unit(i, c8), pack8(&f[8 * x]));
    }
    dg_own += (q4[0] + q4[1]) + (q4[2] + q4[3]);
  }
  {
    const float tot = warp_sum(rho);
    if (lane == 0) red[8 + warp] = tot;  // summed in a fixed order below (deterministic)
  }
  dgo[qd * C + i] = dg_own;
  dbo[qd * C + i] = db_own;
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  if (ok && p.dq32) {
    const size_t row0 = (size_t)(b * p.T + t0) * p.H + h;
    put_wide_tile(p.dq32, Xvn, row0, p.H, p.Dk, imax);
    put_wide_tile(p.dk32, Xdk, row0, p.H, p.Dk, imax);
    put_wide_tile(p.dv32, Xe, row0, p.H, p.Dv, imax);
  } else if (ok && tid == 64) {  // dq, dk and dv leave by tiled stores (rows past the end of the sequence are clipped)
    for (int sl = 0; sl < 2; ++sl) {  // a slab that lies wholly past the true width is not stored at all
      if (64 * sl < p.Dk) {
        tc::tma_store_4d(&maps.dq, tc::smem_u32(Xvn) + 8192 * sl, 64 * sl, h, t0, b);
        tc::tma_store_4d(&maps.dk, tc::smem_u32(Xdk) + 8192 * sl, 64 * sl, h, t0, b);
      }
      if (64 * sl < p.Dv) tc::tma_store_4d(&maps.dv, tc::smem_u32(Xe) + 8192 * sl, 64 * sl, h, t0, b);
    }
    tc::bulk_commit();
  }
  if (tid < 32) {  // dg = reverse cumulative sum of dgam within the chunk: one warp, two rows per lane
    // d/dgam_last: E(gam_last) <dS, S0> and the sum over the rows of k_i . dkp_i
    float base = 0.f, kp = 0.f;
    for (int wv = 0; wv < 8; ++wv) { base += red[wv]; kp += red[8 + wv]; }
    base = L * base + kp;
    const int ra = C - 1 - 2 * tid, rb = ra - 1;
    float a = (dgo[ra] + dgo[C + ra]) + (dgo[2 * C + ra] + dgo[3 * C + ra]);
    float bq = (dgo[rb] + dgo[C + rb]) + (dgo[2 * C + rb] + dgo[3 * C + rb]);
    warp_rcumsum64(a, bq, tid);
    __syncwarp();  // every lane has read its rows before any lane overwrites them
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
  if (warp == 0) tc::tmem_dealloc(tA, 256);
}

// ------------------------------------------------------------------ host
mxb_status tc_run_fwd(TcP& p, cudaStream_t st);
mxb_status tc64_run_bwd(const TcP& p, cudaStream_t st);

// Forward recompute (saving per-chunk states and v_new), reverse state pass, per-chunk pass.
mxb_status tc_run_bwd(TcP& p, bool recompute, cudaStream_t st) {
  p.save = 1;
  mxb_status s = MXB_OK;
  if (recompute) {
    bf16* keep_out = p.out;
    float* keep_hT = p.hT;
    p.out = p.dv;  // the recomputed forward output is not needed; dv is overwritten afterwards
    p.hT = nullptr;
    s = tc_run_fwd(p, st);
    p.out = keep_out;
    p.hT = keep_hT;
    if (s != MXB_OK) return s;
  }
  if (p.Dk == 64 && p.Dv == 64) return tc64_run_bwd(p, st);
  RowMaps maps;
  std::memset(&maps, 0, sizeof maps);
  const bool narrow = p.Dk != KD || p.Dv != KD;  // narrower heads exist only through the copy engine
  const bool tma = (!p.no_tma || narrow) && make_tma_map_bthd(&maps.k, p.k, p.B, p.T, p.H, p.Dk) &&
                   make_tma_map_bthd(&maps.q, p.q, p.B, p.T, p.H, p.Dk) && make_tma_map_bthd(&maps.v, p.v, p.B, p.T, p.H, p.Dv) &&
                   make_tma_map_bthd(&maps.dO, p.dO, p.B, p.T, p.H, p.Dv);
  if (narrow && !tma) return MXB_ERR_UNSUPPORTED;
  auto state = [&](auto tma_v, auto nv) {
    constexpr bool TMA = decltype(tma_v)::value;
    constexpr int NV = decltype(nv)::value;
    if (MXB_ALLOW_SMEM(kStateBwdSmem<NV>, gdn_tc_state_bwd_kernel<TMA, NV>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_tc_state_bwd_kernel", st,
               (launch_kernel(gdn_tc_state_bwd_kernel<TMA, NV>, dim3(p.B * p.H, (p.Dv + NV - 1) / NV), 256, kStateBwdSmem<NV>, st, p, maps)));
    return MXB_OK;
  };
  if (tma && chain_columns(p, true)) s = chain_bwd(p, maps, chain_columns(p, true), st);
  else if (!tma) s = state(std::false_type{}, std::integral_constant<int, KD>{});
  else if (tc_split_columns(p)) s = state(std::true_type{}, std::integral_constant<int, 64>{});
  else s = state(std::true_type{}, std::integral_constant<int, KD>{});
  if (s != MXB_OK) return s;
  s = check_launch("gdn_tc_state_bwd_kernel");
  if (s != MXB_OK) return s;
  // The chunk kernel is fed and drained by the copy engine only (also under MXB_GDN_NO_TMA, which selects the
  // per-thread staging of the kernels that have one): it needs the tensor maps.
  if (!tma) {
    std::memset(&maps, 0, sizeof maps);
    if (!(make_tma_map_bthd(&maps.k, p.k, p.B, p.T, p.H, p.Dk) && make_tma_map_bthd(&maps.q, p.q, p.B, p.T, p.H, p.Dk) &&
          make_tma_map_bthd(&maps.v, p.v, p.B, p.T, p.H, p.Dv) && make_tma_map_bthd(&maps.dO, p.dO, p.B, p.T, p.H, p.Dv)))
      return MXB_ERR_UNSUPPORTED;
  }
  if (!(make_tma_map_bthd(&maps.dq, p.dq, p.B, p.T, p.H, p.Dk) && make_tma_map_bthd(&maps.dk, p.dk, p.B, p.T, p.H, p.Dk) &&
        make_tma_map_bthd(&maps.dv, p.dv, p.B, p.T, p.H, p.Dv)))
    return MXB_ERR_UNSUPPORTED;
  if (MXB_ALLOW_SMEM(kChunkBwdSmem, gdn_tc_chunk_bwd_kernel) != MXB_OK) return MXB_ERR_CUDA;
  MXB_LAUNCH("gdn_tc_chunk_bwd_kernel", st,
             (launch_kernel(gdn_tc_chunk_bwd_kernel, dim3(p.B * p.H, p.n), 256, kChunkBwdSmem, st, p, maps)));
  return check_launch("gdn_tc_chunk_bwd_kernel");
}

}  // namespace mxb
