// Gated delta rule, chunked WY/UT form - tensor-core path (tcgen05.mma, TMEM
// accumulators) for bf16 I/O with fp32 state, chunk 64, Dk and Dv up to 128 (tiles are 128 wide; narrower heads ride
// on the copy engine's zero fill and clipping).
//
// Same mathematics as the fp32 path (gdn_simt.cu; reference
// gated_delta_scan_chunked, gpu/ir.cpp:2352-2550).  Every contraction runs as
// tcgen05.mma.kind::f16 on bf16 operands staged in shared memory (token rows by
// TMA in the 128-byte-swizzled layout, workspace tiles as byte images of the
// canonical layouts of umma_tiles.cuh) with fp32 accumulation in tensor memory;
// the triangular inverse, all decay factors, the recurrent state and every
// reduction stay in fp32.
//
//   gdn_tc_prep_kernel       one CTA per chunk (four per SM): [k;q] k^T (M=128), fp32 solve,
//                            (T beta) v and (T beta) (E(gam) k) (M=64, N=128 each) -> u, w, P, T
//   gdn_tc_state_fwd_kernel  one CTA per (batch, head) and 128 or 64 columns of the state, sequential over
//                            chunks, fp32 state in registers (thread = state row, half of the columns), operands
//                            two chunks ahead: [w;q] S (M=128) -> v_new, then (r k)^T v_new and P v_new
#include <cuda.h>

#include <cstring>

#include "gdn_tc.cuh"

namespace mxb {

// ------------------------------------------------------------------ prep
// u = T (v beta) and w = T (k beta E(gam)) are evaluated as (T diag(beta)) v and
// (T diag(beta)) (diag(E(gam)) k): one column-scaled bf16 copy of T serves both, k, q and v are staged raw
// and k is scaled in place while T is formed.
//
// A CTA is a chain of dependent steps (copy -> MMA -> epilogue -> solve -> MMA -> epilogue -> stores) that leaves
// the SM idle most of the time, so the kernel is sized for FOUR CTAs per SM: 128 TMEM columns (u and w side by side,
// 64 each, once the product before has been read) and 51 KB of shared memory, every region reused as soon as it is dead:
//   [k;q] (32 KB, two slabs of 64 columns: k box then q box)  ->  v lands in the q boxes once q k^T is done
//                                                              ->  k scaled to diag(d) k in place during the solve
//                                                              ->  u image over v, w image over k
//   A / T fp32 matrix (17 KB): then the bf16 T image on its way out and T diag(beta), the one operand of both
//   products (w = (T diag beta)(diag(d) k)), over it
//   P goes from the accumulator straight to the workspace (a warp's stores fill whole 128-byte lines of the image)
// TMA = true: k, q, v arrive as cp.async.bulk.tensor tiles (boxes of 64 rows x 64 columns, 128-byte
// swizzle; rows past the end of the sequence are zero-filled by the copy engine).  TMA = false: the same
// tiles staged with cp.async into the same swizzled positions (kept as a cross-check and for drivers
// without the tensor-map entry point).
constexpr int kPrepSmem = 32768 + C * LDA * 4 + 3 * C * 4 + 64 + 64 + 1024;
static_assert(C * LDA * 4 >= 2 * 8192, "the T image and T diag(beta) go over the fp32 matrix");
static_assert(4 * (kPrepSmem + 1024) <= 228 * 1024, "four CTAs per SM");

using PrepMaps = RowMaps;


template <bool TMA>
__global__ void __launch_bounds__(128, 4) gdn_tc_prep_kernel(TcP p, const __grid_constant__ PrepMaps maps) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Akq = sm;                    // slab s at 16384 s: k box [64][64], then q box [64][64] (later v, u / w images)
  float* Am = reinterpret_cast<float*>(Akq + 32768);  // [64][LDA]  A, then T in place
  uint8_t* Tt = reinterpret_cast<uint8_t*>(Am);       // [64 i][64 m] T image, over the fp32 matrix once it is dead
  uint8_t* Tb = Tt + 8192;              // [64 i][64 m] T diag(beta), behind it
  float* gam = Am + C * LDA;
  float* bet = gam + C;
  float* dd = bet + C;                  // E(gam)
  uint64_t* mbar = reinterpret_cast<uint64_t*>(dd + C);  // [0] MMA completion, [1] k,q landed, [2] v landed
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 4);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H, t0 = c * C;
  const size_t ci = (size_t)bh * p.n + c;
  auto row = [&](int i) { return ((size_t)(b * p.T + t0 + i) * p.H + h); };
  const int imax = min(C, p.T - t0);
  const uint32_t sAkq = tc::smem_u32(Akq);
  // byte offset in Akq of unit (i, c8) of the k tile; the q (later v) tile sits 8192 bytes further
  auto kq_unit = [](int i, int c8) {
    return (uint32_t)(c8 >> 3) * 16384u + (uint32_t)i * 128u + (uint32_t)(((c8 & 7) ^ (i & 7)) << 4);
  };

  // The first CTA clears the status header: whoever raises it has waited in vain for far longer than this takes.
  if (c == 0 && bh == 0 && tid < 64) p.status[tid] = 0;
  // prologue latencies side by side: warp 0 allocates TMEM, warp 1 reads the gates, one thread of warp 2
  // initialises the barriers and issues the copies that complete on them
  if (tid == 64) {
    tc::mbar_init(&mbar[0], 1);
    tc::mbar_init(&mbar[1], 1);
    tc::mbar_init(&mbar[2], 1);
    tc::mbar_fence_init();
  }
  if (TMA) {
    if (tid == 64) {
      tc::mbar_expect_tx(&mbar[1], 32768);
      for (int sl = 0; sl < 2; ++sl) {
        tc::tma_load_4d(sAkq + sl * 16384, &maps.k, 64 * sl, h, t0, b, &mbar[1]);
        tc::tma_load_4d(sAkq + sl * 16384 + 8192, &maps.q, 64 * sl, h, t0, b, &mbar[1]);
      }
    }
  } else {
    for (int u = tid; u < 64 * 16; u += 128) {
      const int i = urow16(u), c8 = ucol16(u);
      const bool ok = i < imax;
      const size_t g = ok ? row(i) * KD + c8 * 8 : 0;
      tc::cp_async16(sAkq + kq_unit(i, c8), p.k + g, ok);
      tc::cp_async16(sAkq + 8192 + kq_unit(i, c8), p.q + g, ok);
    }
    tc::cp_async_commit();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, 128);
    tc::tmem_relinquish();
  }
  if (warp == 1) {  // in-chunk inclusive cumulative sum of the log gate: two elements per lane
    const bool ok0 = 2 * lane < imax, ok1 = 2 * lane + 1 < imax;
    const float g0 = ok0 ? log_gate_tc(p.gate[row(2 * lane)], p.gate_is_log) : 0.f;
    const float g1 = ok1 ? log_gate_tc(p.gate[row(2 * lane + 1)], p.gate_is_log) : 0.f;
    float s = g0 + g1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    const float c1 = s, c0 = s - g1;
    const float b0 = ok0 ? p.beta[row(2 * lane)] : 0.f, b1 = ok1 ? p.beta[row(2 * lane + 1)] : 0.f;
    gam[2 * lane] = c0; gam[2 * lane + 1] = c1;
    bet[2 * lane] = b0; bet[2 * lane + 1] = b1;
    dd[2 * lane] = exp_nonpos(c0); dd[2 * lane + 1] = exp_nonpos(c1);
    p.gam[ci * C + 2 * lane] = c0;
    p.gam[ci * C + 2 * lane + 1] = c1;
  }
  bool ok = true;
  if (TMA) {
    __syncthreads();  // barriers initialised before anyone waits on them
    ok = tc::mbar_wait(&mbar[1], 0);  // [k;q]
  } else {
    tc::cp_async_wait<0>();
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  // D0[128 x 64] = [k;q] k^T
  if (tid == 0) {
    const tc::Tile a = tc::kmajor_sw128_tile(Akq, 16384);
    tc::issue_gemm(taddr, a, a, 128, 64, KD, false);  // B = first 64 rows of the same tile
    tc::mma_commit(mbar);
  }
  if (ok) ok = tc::mbar_wait(mbar, 0);
  tc::fence_after_sync();
  // q is dead: v takes its place (needed only for the second MMA, long after the solve)
  if (TMA) {
    if (tid == 64) {
      tc::mbar_expect_tx(&mbar[2], 16384);
      for (int sl = 0; sl < 2; ++sl) tc::tma_load_4d(sAkq + sl * 16384 + 8192, &maps.v, 64 * sl, h, t0, b, &mbar[2]);
    }
  } else {
    for (int u = tid; u < 64 * 16; u += 128) {
      const int i = urow16(u), c8 = ucol16(u);
      const bool okv = i < imax;
      tc::cp_async16(sAkq + 8192 + kq_unit(i, c8), okv ? p.v + row(i) * KD + c8 * 8 : p.v, okv);
    }
    tc::cp_async_commit();
  }
  if (ok) {
    const int i = tid & 63;
    const float gi = gam[i], bi = bet[i];
    for (int c0 = 0; c0 < 64; c0 += 32) {
      float f[32];
      ld_acc32(taddr, warp, c0, f);
      if (tid < 64) {  // A = -(k beta k^T) Gamma, strictly lower
        // all 32 values first, then the stores: a store into A between the loads of gam would pin the order
        // (the compiler must assume the two shared arrays overlap) and the exponentials would run one by one
#pragma unroll
        for (int jj = 0; jj < 32; ++jj) {
          const int j = c0 + jj;
          const float val = -bi * f[jj] * exp_nonpos(gi - gam[j]);
          f[jj] = (j < i) ? val : 0.f;
        }
#pragma unroll
        for (int x = 0; x < 8; ++x)
          *reinterpret_cast<float4*>(Am + i * LDA + c0 + 4 * x) = make_float4(f[4 * x], f[4 * x + 1], f[4 * x + 2], f[4 * x + 3]);
      } else {         // P = (q k^T) Gamma, lower incl. diagonal -> straight into its operand-tile image in the workspace
        uint32_t pk[16];
#pragma unroll
        for (int jj = 0; jj < 32; jj += 2) {
          const int j = c0 + jj;
          const float v0 = f[jj] * exp_nonpos(gi - gam[j]), v1 = f[jj + 1] * exp_nonpos(gi - gam[j + 1]);
          const float x0 = (j <= i) ? v0 : 0.f, x1 = (j + 1 <= i) ? v1 : 0.f;
          pk[jj >> 1] = tc::pack_bf16(x0, x1);
        }
        uint8_t* pimg = reinterpret_cast<uint8_t*>(p.P + ci * C * C);
#pragma unroll
        for (int x = 0; x < 4; ++x)  // eight consecutive rows of a unit column are one 128-byte line of the image
          *reinterpret_cast<uint4*>(pimg + tc::kmajor_unit(i, (c0 >> 3) + x, C)) =
              make_uint4(pk[4 * x], pk[4 * x + 1], pk[4 * x + 2], pk[4 * x + 3]);
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // The other half of the CTA meanwhile turns k into diag(d) k in place (its product with itself is done), so that
  // w = (T diag beta)(diag(d) k) needs no second scaled copy of T.
  invert_unit_lower(Am, ok, [&](int i) {
    const float di = dd[i];
#pragma unroll
    for (int c8 = 0; c8 < 16; ++c8) {
      uint4* unit = reinterpret_cast<uint4*>(Akq + kq_unit(i, c8));
      *unit = tc::scale_bf16x8(*unit, di);
    }
  });
  {  // the T image and the bf16 operand tile T diag(beta) go over the fp32 matrix: read everything, barrier, write
    uint4 timg[4], tbimg[4];
    load_inverse_images(Am, bet, timg, tbimg);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      sts16(Tt, 16 * (tid + 128 * m), timg[m]);
      sts16(Tb, 16 * (tid + 128 * m), tbimg[m]);
    }
  }
  if (TMA) { if (ok) ok = tc::mbar_wait(&mbar[2], 0); }  // v
  else tc::cp_async_wait<0>();
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // u = (T beta) v and w = (T beta)(d k), contracted over the rows of v and k; weight-stationary: a thread has a row and
  // half of the columns of both
  if (ok && tid == 0) {
    tc::issue_gemm<true>(taddr, tc::kmajor_tile(Tb, C), tc::mnmajor_sw128_tile(Akq + 8192, 16384), 64, KD, C, false);
    tc::issue_gemm<true>(taddr + 64, tc::kmajor_tile(Tb, C), tc::mnmajor_sw128_tile(Akq, 16384), 64, KD, C, false);
    tc::mma_commit(mbar);
    tc::bulk_store(p.Tm + ci * C * C, tc::smem_u32(Tt), 8192);  // T leaves as the byte image of its operand tile
    tc::bulk_commit();
  }
  if (ok) ok = tc::mbar_wait(mbar, 1);
  tc::fence_after_sync();
  if (ok) {
    // the u image (column-blocked: columns 0-63 and 64-127 are its two contiguous halves) over the v boxes, and the w image
    // in the 128-byte-swizzled layout of a TMA tile (two 8 KB slabs of 64 columns) over the k boxes, so that the state
    // kernels can put it beside TMA-loaded q rows in one operand
    const int ir = 32 * (warp & 1) + lane, c8 = 8 * (warp >> 1);
#pragma unroll
    for (int c0 = 0; c0 < 64; c0 += 32) {
      float f[32];
      ld_acc32(taddr, warp, c0, f);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const uint32_t off = tc::colblk_unit(ir, c8 + (c0 >> 3) + x, C);
        sts16(Akq, 8192u + (off >> 13) * 16384u + (off & 8191u), pack8(&f[8 * x]));
      }
      ld_acc32(taddr + 64, warp, c0, f);
#pragma unroll
      for (int x = 0; x < 4; ++x) sts16(Akq, kq_unit(ir, c8 + (c0 >> 3) + x), pack8(&f[8 * x]));
    }
  } else if (tid == 0) {
    atomicExch(p.status, 1);
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  if (tid == 0) {
    if (ok) {
      for (int hf = 0; hf < 2; ++hf) {
        tc::bulk_store(p.u + ci * C * KD + hf * 4096, sAkq + 8192 + hf * 16384, 8192);
        tc::bulk_store(p.w + ci * C * KD + hf * 4096, sAkq + hf * 16384, 8192);
      }
      tc::bulk_commit();
    }
    tc::bulk_wait_read<0>();  // shared memory must outlive the copies
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 128);
}

// ------------------------------------------------------------ state forward
// One CTA (256 threads) per (batch, head) and NV columns.  Thread t owns state row kk = t & 127 and the
// columns of half t >> 7.  The operand tiles are buffered (buffer c & 1 for chunk c; k: c % 3) and requested as soon
// as the MMA (or epilogue) that last read the buffer has finished, a chunk period or more before they are needed:
//   A  [w;q]   buffer free after w S           needed before w S
//   U  u       free after v_new                needed before v_new
//   K  k       free after (r k)^T v_new        needed in the shadow of the chunk before (k is scaled in place there)
//   P          free after P v_new              needed before P v_new
//
// Bound by the chain S -> w S -> v_new -> (r k)^T v_new -> S where the heads are few, by HBM where they fill the GPU.
// Only what the chain needs stands between its products: q S and the output rows (E(gam) q S + P v_new) are finished in
// the shadow of the next chunk's w S, the decay factors and the scaled k of the next chunk in the shadow of this one's
// products, and P v_new is issued behind the state update (16 heads of 128, 24 chunks, NV = 64: 2.3 -> 1.9 us a chunk).  More work moved into the shadow of w S
// (half of the scaling of k, the u operand into registers) slowed the product down: both need shared memory, 47 -> 50 us.
//
// TMA = true: q and k rows arrive as tensor-map boxes (128-byte swizzle) issued by ONE thread and complete on the
// barrier of their group, like the images: no thread spends issue slots on copies (four cp.async per thread and
// group cost every thread ~1.6 k and ~1.1 k cycles per chunk).
// TMA = false: the same rows by cp.async into the same swizzled positions.
//
// NV: columns of the state per CTA.  128 (all of them) where the (batch, head) pairs fill the GPU; 64 otherwise: a
// chunk's chain of products and epilogues is then half as wide (columns of the state are independent; w, q, k and P are
// read by both CTAs, the second time from L2).
template <int NV>
constexpr int kStateFwdSmem =
    2 * 32768 + 256 * NV + 2 * 8192 + 128 * NV + 128 * NV + 3 * 16384 + 2 * 128 * NV + 4 * C * 4 + 128 + 1024;

template <bool TMA, int NV>
__global__ void __launch_bounds__(kStateThreads<NV>, 1) gdn_tc_state_fwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  static_assert(NV == KD || TMA, "the per-thread staging moves whole rows");
  constexpr int NC = NV / 2;                   // columns per thread
  const int col0 = blockIdx.y * NV;
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* A1 = sm;                 // x2 [128: w rows 0-63, q rows 64-127][128 kk], two swizzled slabs of 64 columns
  uint8_t* Sop = A1 + 2 * 32768;    // [128 kk][NV j]    bf16 copy of the state
  uint8_t* Pm = Sop + 256 * NV;     // x2 [64 i][64 m]   P
  uint8_t* Vn = Pm + 2 * 8192;      // [64 i][NV j]      v_new
  uint8_t* Ot = Vn + 128 * NV;      // [64 i][NV j]      output tile on its way out (swizzled slabs of 64 columns)
  uint8_t* A3 = Ot + 128 * NV;      // x3 [64 i][128 kk] k, then diag(E(gam_last-gam_i)) k  (A = k^T), swizzled slabs
  uint8_t* Ut = A3 + 3 * 16384;     // x2 [64 i][NV j]   u
  float* dd = reinterpret_cast<float*>(Ut + 2 * 128 * NV);
  float* rr = dd + 2 * C;           // (both: two buffers)
  // [0] w S and q S, later (r k)^T v_new; [10] P v_new; landed, per buffer: [1..] w image and q rows, [3..] u image,
  // [5..] k rows, [8..] P image
  uint64_t* mbar = reinterpret_cast<uint64_t*>(rr + 2 * C);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 11);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int kk = tid & 127, half = tid >> 7, j0 = NC * half;  // (of the 256 threads of warps 0-7)
  auto lead = [&] { return warp == 8 && tc::elect_one(); };  // issues the products and the copies
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
  const uint32_t sA1b = tc::smem_u32(A1), sPb = tc::smem_u32(Pm), sA3b = tc::smem_u32(A3), sUb = tc::smem_u32(Ut);
  const uint32_t sOt = tc::smem_u32(Ot);

  auto grow = [&](int c, int i) { return ((size_t)(b * p.T + c * C + i) * p.H + h); };
  // The workspace tiles (w, u, P) are byte images of the operand layout: one bulk copy each, completing on an mbarrier.
  // Slab s of A1 (columns 64 s ..): the w slab (rows 0-63), then the q box (rows 64-127).
  auto load_A = [&](int c) {  // [w;q] of chunk c
    if (c >= p.n) return;
    const size_t ci = (size_t)bh * p.n + c;
    const uint32_t sA1 = sA1b + (c & 1) * 32768;
    uint64_t* mb = &mbar[1 + (c & 1)];
    tc::mbar_expect_tx(mb, TMA ? 32768 : 16384);
    for (int sl = 0; sl < 2; ++sl) {
      tc::bulk_load(sA1 + sl * 16384, p.w + ci * C * KD + sl * 4096, 8192, mb);
      if (TMA) tc::tma_load_4d(sA1 + sl * 16384 + 8192, &maps.q, 64 * sl, h, c * C, b, mb);
    }
  };
  auto load_U = [&](int c) {
    if (c >= p.n) return;
    uint64_t* mb = &mbar[3 + (c & 1)];
    tc::mbar_expect_tx(mb, 128 * NV);
    tc::bulk_load(sUb + (c & 1) * 128 * NV, p.u + ((size_t)bh * p.n + c) * C * KD + C * col0, 128 * NV, mb);
  };
  auto load_K = [&](int c) {
    if (!TMA || c >= p.n) return;
    uint64_t* mb = &mbar[5 + c % 3];
    tc::mbar_expect_tx(mb, 16384);
    for (int sl = 0; sl < 2; ++sl) tc::tma_load_4d(sA3b + (c % 3) * 16384 + sl * 8192, &maps.k, 64 * sl, h, c * C, b, mb);
  };
  auto load_P = [&](int c) {
    if (c >= p.n) return;
    tc::mbar_expect_tx(&mbar[8 + (c & 1)], 8192);
    tc::bulk_load(sPb + (c & 1) * 8192, p.P + ((size_t)bh * p.n + c) * C * C, 8192, &mbar[8 + (c & 1)]);
  };
  auto store_out = [&](int c) {
    for (int sl = 0; sl < (TMA && !p.out32 ? NV / 64 : 0); ++sl)  // a slab that lies wholly past the true width is not stored at all
      if (col0 + 64 * sl < p.Dv) tc::tma_store_4d(&maps.o, sOt + sl * 8192, col0 + 64 * sl, h, c * C, b);
  };
  // TMA = false: the q and k rows, by the 256 threads (a group per call, empty past the end)
  auto copy_q = [&](int c) {
    if (TMA) return;
    const int imax = c < p.n ? min(C, p.T - c * C) : -1;
    for (int u = tid; u < 64 * 16 && imax >= 0; u += 256) {
      const int i = urow16(u), c8 = ucol16(u);
      const uint32_t off = (uint32_t)(c8 >> 3) * 16384u + 8192u + (uint32_t)i * 128u + (uint32_t)(((c8 & 7) ^ (i & 7)) << 4);
      tc::cp_async16(sA1b + (c & 1) * 32768 + off, i < imax ? p.q + grow(c, i) * KD + c8 * 8 : p.q, i < imax);
    }
    tc::cp_async_commit();
  };
  auto copy_k = [&](int c) {
    if (TMA) return;
    const int imax = c < p.n ? min(C, p.T - c * C) : -1;
    for (int u = tid; u < 64 * 16 && imax >= 0; u += 256) {
      const int i = urow16(u), c8 = ucol16(u);
      tc::cp_async16(sA3b + (c % 3) * 16384 + tc::sw128_unit(i, c8), i < imax ? p.k + grow(c, i) * KD + c8 * 8 : p.k, i < imax);
    }
    tc::cp_async_commit();
  };

  if (warp == 0) {
    tc::tmem_alloc(tslot, 512);
    tc::tmem_relinquish();
  }
  if (lead()) {
    for (int m = 0; m < 11; ++m) tc::mbar_init(&mbar[m], 1);
    tc::mbar_fence_init();
    for (int c = 0; c < 2; ++c) {
      load_A(c);
      load_U(c);
      load_K(c);
      load_P(c);
    }
    load_K(2);
  }
  if (warp >= 8) {
    if (NV == KD) tc::reg_dec<40>();
    tc::fence_before_sync();
    __syncthreads();  // barriers initialised, TMEM allocated
    tc::fence_after_sync();
    const uint32_t taddr = *tslot;
    uint32_t ph = 0;
    bool ok = true;
    for (int c = 0; c < p.n; ++c) {
      const size_t ci = (size_t)bh * p.n + c;
      const int buf = c & 1;
      const uint32_t lph = (c >> 1) & 1;  // phase of the image barriers of this buffer
      if (lead()) {
        tc::bulk_wait_read<0>();  // v_new and the output tile of the chunk before have left
        ok = tc::mbar_wait(&mbar[1 + buf], lph);
      }
      ok = __syncthreads_and(ok);
      if (!ok) break;
      if (lead()) {
        tc::fence_after_sync();
        // D1 = [w;q] S
        tc::issue_gemm(taddr, tc::kmajor_sw128_tile(A1 + buf * 32768, 16384), tc::colblk_mnmajor_tile(Sop, KD), 128, NV, KD, false);
        tc::mma_commit(mbar);
        if (p.save) {  // the state at chunk start, saved for the backward as the byte image of the operand tile
          tc::bulk_store(p.hs + ci * KD * KD + KD * col0, tc::smem_u32(Sop), 256 * NV);
          tc::bulk_commit();
        }
        if (c > 0) {
          ok = tc::mbar_wait(&mbar[10], (c - 1) & 1);
          if (ok) load_P(c + 1);
        }
        ok = ok && tc::mbar_wait(&mbar[8 + buf], lph);
        ok = ok && tc::mbar_wait(mbar, ph);
        if (ok) load_A(c + 2);
        tc::bulk_wait_read<0>();  // the state image has left its tile
      }
      ph ^= 1;
      __syncthreads();
      if (lead() && ok) {
        tc::fence_after_sync();
        // D3 = (r k)^T v_new, which the next chunk waits for, then P v_new into rows 64-127 of D2: the tile is the 128 rows
        // that end with P; what the 64 rows before it hold (other tiles) only reaches rows of D2 that nothing reads
        tc::issue_gemm(taddr + 256, tc::mnmajor_sw128_tile(A3 + (c % 3) * 16384, 8192), tc::colblk_mnmajor_tile(Vn, C), 128, NV, C, false);
        tc::mma_commit(mbar);
        tc::issue_gemm(taddr + 128, tc::kmajor_tile(Pm + (buf - 1) * 8192, C), tc::colblk_mnmajor_tile(Vn, C), 128, NV, C, false);
        tc::mma_commit(mbar + 10);
        if (p.save) tc::bulk_store(p.vn + ci * C * KD + C * col0, tc::smem_u32(Vn), 128 * NV);
        if (c > 0) store_out(c - 1);  // (its tile is complete since the barrier above)
        tc::bulk_commit();
        load_U(c + 2);  // u has been consumed by every thread
        ok = tc::mbar_wait(mbar, ph);
        if (ok) load_K(c + 3);
      }
      ph ^= 1;
    }
    if (lead()) tc::bulk_wait_read<0>();
    __syncthreads();  // the output tile is free
    __syncthreads();  // and full
    if (lead()) {
      if (ok) {
        store_out(p.n - 1);
        tc::bulk_commit();
      } else {
        atomicExch(p.status, 2);
      }
      tc::bulk_wait_read<0>();  // shared memory must outlive the copies
    }
    __syncthreads();
    return;
  }
  if (NV == KD) tc::reg_inc<216>();
  copy_q(0);
  copy_k(0);
  copy_q(1);
  copy_k(1);
  copy_k(2);
  float S[NC];  // state row kk, columns col0 + j0 .. (zero outside the true Dk x Dv state)
  if (p.h0) {
    const float4* src = reinterpret_cast<const float4*>(p.h0 + ((size_t)bh * p.Dk + kk) * p.Dv + col0 + j0);
#pragma unroll
    for (int x = 0; x < NC / 4; ++x) {
      const float4 t4 = (kk < p.Dk && col0 + j0 + 4 * x < p.Dv) ? __ldg(src + x) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[4 * x] = t4.x; S[4 * x + 1] = t4.y; S[4 * x + 2] = t4.z; S[4 * x + 3] = t4.w;
    }
  } else {
#pragma unroll
    for (int x = 0; x < NC; ++x) S[x] = 0.f;
  }
  // Decay factors of a chunk, fetched and computed while the tensor core works on the chunk before it; the k rows of a
  // chunk are scaled by r in place there too, so that the state update contracts them with v_new itself (every thread
  // scales the 16-byte units it would copy in the cp.async variant: no barrier needed for those).
  float g_nxt = p.gam[(size_t)bh * p.n * C + (tid & 63)], gl_nxt = p.gam[(size_t)bh * p.n * C + C - 1];
  auto decay = [&](int c) {
    if (tid < C) {
      dd[(c & 1) * C + tid] = exp_nonpos(g_nxt);
      rr[(c & 1) * C + tid] = exp_nonpos(gl_nxt - g_nxt);
    }
  };
  bool ok = true;
  auto scale_k = [&](int c) {
    if (TMA && ok) ok = tc::mbar_wait(&mbar[5 + c % 3], (c / 3) & 1);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int u = tid + 256 * m, i = urow16(u);
      uint4* unit = reinterpret_cast<uint4*>(A3 + (c % 3) * 16384 + tc::sw128_unit(i, ucol16(u)));
      *unit = tc::scale_bf16x8(*unit, rr[(c & 1) * C + i]);
    }
  };
  decay(0);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  if (!TMA) tc::cp_async_wait<3>();  // k of chunk 0 (groups q0 k0 q1 k1 k2)
  scale_k(0);
  uint32_t ph = 0;
  float f[NC];  // accumulator row; rows 64-127 keep E(gam_i) (q S) here until P v_new arrives
  // out = E(gam)(q S) + P v_new of chunk c, rows in the upper half of the threads
  auto put_out = [&](int c) {
    if (ok) ok = tc::mbar_wait(&mbar[10], c & 1);
    tc::fence_after_sync();
    if (!ok || kk < 64) return;  // (warp-uniform)
    const int i = kk & 63;
    float a[NC];
    ld_accN(taddr + 128 + j0, warp, a);
    uint4 o[NC / 8];
#pragma unroll
    for (int x = 0; x < NC / 8; ++x)
      o[x] = make_uint4(tc::pack_bf16(f[8 * x] + a[8 * x], f[8 * x + 1] + a[8 * x + 1]),
                        tc::pack_bf16(f[8 * x + 2] + a[8 * x + 2], f[8 * x + 3] + a[8 * x + 3]),
                        tc::pack_bf16(f[8 * x + 4] + a[8 * x + 4], f[8 * x + 5] + a[8 * x + 5]),
                        tc::pack_bf16(f[8 * x + 6] + a[8 * x + 6], f[8 * x + 7] + a[8 * x + 7]));
    if (p.out32) {
      if (c * C + i < p.T) {
        float* dst = p.out32 + grow(c, i) * p.Dv + col0 + j0;
#pragma unroll
        for (int x = 0; x < NC / 8; ++x)
          if (col0 + j0 + 8 * x < p.Dv) put_wide(dst + 8 * x, o[x]);
      }
    } else if (TMA) {  // into the swizzled output tile; one thread hands it to the copy engine after the next barrier
#pragma unroll
      for (int x = 0; x < NC / 8; ++x) sts16(Ot, tc::sw128_unit(i, NC / 8 * half + x), o[x]);
    } else if (c * C + i < p.T) {
      uint4* dst = reinterpret_cast<uint4*>(p.out + grow(c, i) * KD + j0);
#pragma unroll
      for (int x = 0; x < NC / 8; ++x) dst[x] = o[x];
    }
  };
  for (int c = 0; c < p.n; ++c) {
    const size_t ci = (size_t)bh * p.n + c;
    const int buf = c & 1;
    const uint32_t lph = (c >> 1) & 1;  // phase of the image barriers of this buffer
    const float L = exp_nonpos(gl_nxt);
    if (c + 1 < p.n) {
      g_nxt = p.gam[(ci + 1) * C + (tid & 63)];
      gl_nxt = p.gam[(ci + 1) * C + C - 1];
    }
#pragma unroll
    for (int c8 = 0; c8 < NC / 8; ++c8) {  // state as the MMA operand (and saved for the backward)
      const uint4 val = make_uint4(tc::pack_bf16(S[8 * c8], S[8 * c8 + 1]), tc::pack_bf16(S[8 * c8 + 2], S[8 * c8 + 3]),
                                   tc::pack_bf16(S[8 * c8 + 4], S[8 * c8 + 5]), tc::pack_bf16(S[8 * c8 + 6], S[8 * c8 + 7]));
      sts16(Sop, tc::colblk_unit(kk, NC / 8 * half + c8, KD), val);
    }
    if (!TMA) tc::cp_async_wait<3>();  // q rows of this chunk (groups since: k of it, q and k of the next, k of the third)
    tc::fence_async_smem();
    tc::fence_before_sync();
    ok = __syncthreads_and(ok);  // the barrier also makes the verdict of the bounded waits uniform, so that all
    if (!ok) break;              // threads leave the loop together
    tc::fence_after_sync();
    // in the shadow of [w;q] S: the output of the chunk before, the decay factors of the chunk after
    if (c > 0) put_out(c - 1);
    decay(c + 1);
    if (ok) ok = tc::mbar_wait(&mbar[3 + buf], lph);  // u image of this chunk
    if (ok) ok = tc::mbar_wait(mbar, ph);
    ph ^= 1;
    tc::fence_after_sync();
    copy_q(c + 2);
    if (ok) {
      const int i = kk & 63;
      ld_accN(taddr + j0, warp, f);
      if (kk < 64) {  // v_new = u - w S
#pragma unroll
        for (int x = 0; x < NC / 8; ++x) {
          const int c8 = NC / 8 * half + x;
          const uint4 uu = *reinterpret_cast<const uint4*>(Ut + buf * 128 * NV + tc::colblk_unit(i, c8, C));
          float e[8];
          tc::unpack_bf16(uu.x, e[0], e[1]); tc::unpack_bf16(uu.y, e[2], e[3]);
          tc::unpack_bf16(uu.z, e[4], e[5]); tc::unpack_bf16(uu.w, e[6], e[7]);
#pragma unroll
          for (int y = 0; y < 8; ++y) e[y] -= f[8 * x + y];
          sts16(Vn, tc::colblk_unit(i, c8, C), make_uint4(tc::pack_bf16(e[0], e[1]), tc::pack_bf16(e[2], e[3]),
                                                          tc::pack_bf16(e[4], e[5]), tc::pack_bf16(e[6], e[7])));
        }
      } else {
        const float di = dd[buf * C + i];
#pragma unroll
        for (int jj = 0; jj < NC; ++jj) f[jj] *= di;
      }
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    if (c + 1 < p.n) {
      if (!TMA) tc::cp_async_wait<2>();  // k of the next chunk (groups since: k of the third, q of the third)
      scale_k(c + 1);
    }
    if (ok) {
      ok = tc::mbar_wait(mbar, ph);
      ph ^= 1;
    }
    tc::fence_after_sync();
    copy_k(c + 3);
    if (ok) {
      float a[NC];
      ld_accN(taddr + 256 + j0, warp, a);  // S <- E(gam_last) S + (r k)^T v_new
#pragma unroll
      for (int jj = 0; jj < NC; ++jj) S[jj] = fmaf(L, S[jj], a[jj]);
    }
    tc::fence_before_sync();
  }
  __syncthreads();  // the output tile is free
  put_out(p.n - 1);
  tc::fence_async_smem();
  __syncthreads();
  if (!ok && tid == 0) atomicExch(p.status, 2);
  if (ok && p.hT && kk < p.Dk) {
    float4* dst = reinterpret_cast<float4*>(p.hT + ((size_t)bh * p.Dk + kk) * p.Dv + col0 + j0);
#pragma unroll
    for (int x = 0; x < NC / 4; ++x)
      if (col0 + j0 + 4 * x < p.Dv) dst[x] = make_float4(S[4 * x], S[4 * x + 1], S[4 * x + 2], S[4 * x + 3]);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 512);
}

// ------------------------------------------------------------------ host
size_t gdn_simt_workspace_bytes(const mxb_gdn_desc* d, bool bwd);
mxb_status gdn_simt_bwd(const mxb_gdn_desc*, const void*, const void*, const void*, const float*,
                        const float*, const float*, const void*, const float*, void*, void*, void*,
                        float*, float*, float*, void*, cudaStream_t);

// chunk > 64 is computed with chunks of 64 (the result does not depend on the chunk size).  Heads narrower than the
// 128-wide tiles (64 <= Dk, Dv < 128, multiples of 8 so that rows stay 16-byte aligned) use the same kernels: their
// tensor maps carry the true width, loads of the missing columns return zeros and stores of them are clipped.
bool gdn_tc_supported(const mxb_gdn_desc* d) {
  auto width_ok = [](int w) { return w >= 64 && w <= KD && w % 8 == 0; };
  return d->io_dtype == MXB_BF16 && width_ok(d->Dk) && width_ok(d->Dv) && d->chunk >= C;
}

// Heads of exactly 64 columns have kernels of their own (gdn_tc64.cu); every other width up to 128 rides on 128-wide tiles.
static bool is64(const TcP& p) { return p.Dk == 64 && p.Dv == 64; }

static size_t carve_tc(TcP& p, void* ws, bool bwd) {
  Carver cv(ws);
  const size_t nc = (size_t)p.B * p.H * p.n, KD = is64(p) ? 64 : tcg::KD;  // width of the tiles
  p.status = cv.take<int>(64);
  p.gam = cv.take<float>(nc * C);
  p.Tm = cv.take<bf16>(nc * C * C);
  p.w = cv.take<bf16>(nc * C * KD);
  p.u = cv.take<bf16>(nc * C * KD);
  p.P = cv.take<bf16>(nc * C * C);
  if (is64(p)) p.Pt = cv.take<bf16>(nc * C * C);
  if (bwd) {
    p.hs = cv.take<bf16>(nc * KD * KD);
    p.vn = cv.take<bf16>(nc * C * KD);
    p.dhs = cv.take<bf16>(nc * KD * KD);
    p.dvn = cv.take<bf16>(nc * C * KD);
  }
  return cv.bytes();
}

static TcP make_tc(const mxb_gdn_desc* d) {
  TcP p{};
  p.B = d->B; p.T = d->T; p.H = d->H;
  p.Dk = d->Dk; p.Dv = d->Dv;
  p.n = (d->T + C - 1) / C;
  p.gate_is_log = d->gate_is_log;
  return p;
}

size_t gdn_tc_workspace_bytes(const mxb_gdn_desc* d, bool bwd) {
  TcP p = make_tc(d);
  const size_t own = carve_tc(p, nullptr, bwd);
  if (!bwd) return own;
  const size_t simt = gdn_simt_workspace_bytes(d, true);
  return own > simt ? own : simt;
}

mxb_status tc_run_bwd(TcP& p, bool recompute, cudaStream_t st);
mxb_status tc64_run_fwd(TcP& p, cudaStream_t st);

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}
// [B,T,H,D] bf16 as a 4-d tensor (D, H, T, B) with boxes of 64 columns x 64 time steps, 128-byte swizzle
// (D a multiple of 8: rows are 16-byte multiples; columns past D and rows past T are zero-filled by the copy engine
// on loads and clipped on stores); float32 tensors: boxes of 32 columns.  Shared with the other kernels.
static bool make_tma_map(CUtensorMap* m, CUtensorMapDataType type, int size, const void* base, int B, int T, int H, int D, int cols = 0) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn || (reinterpret_cast<uintptr_t>(base) & 15) || D * size % 16 || D <= 0) return false;
  const cuuint64_t row = (cuuint64_t)D * size;
  const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)T, (cuuint64_t)B};
  const cuuint64_t strides[3] = {row, H * row, T * (H * row)};
  const cuuint32_t box[4] = {cols ? (cuuint32_t)cols : 128u / size, 1, 64, 1}, estr[4] = {1, 1, 1, 1};
  const CUtensorMapSwizzle swizzle = box[0] * size == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                                     : box[0] * size == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                           : CU_TENSOR_MAP_SWIZZLE_32B;
  return fn(m, type, 4, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool make_tma_map_bthd(CUtensorMap* m, const void* base, int B, int T, int H, int D) {
  return make_tma_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, B, T, H, D);
}
bool make_tma_map_cols(CUtensorMap* m, const void* base, int B, int T, int H, int D, int cols) {
  return make_tma_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, B, T, H, D, cols);
}
bool make_tma_map_f32(CUtensorMap* m, const void* base, int B, int T, int H, int D) {
  return make_tma_map(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, B, T, H, D);
}

mxb_status tc_run_fwd(TcP& p, cudaStream_t st) {
  if (is64(p)) return tc64_run_fwd(p, st);
  PrepMaps maps;
  std::memset(&maps, 0, sizeof maps);
  // heads narrower than the tiles exist only through the copy engine (the per-thread staging addresses full rows)
  const bool narrow = p.Dk != KD || p.Dv != KD;
  const bool tma = (!p.no_tma || narrow) && make_tma_map_bthd(&maps.k, p.k, p.B, p.T, p.H, p.Dk) &&
                   make_tma_map_bthd(&maps.q, p.q, p.B, p.T, p.H, p.Dk) && make_tma_map_bthd(&maps.v, p.v, p.B, p.T, p.H, p.Dv) &&
                   make_tma_map_bthd(&maps.o, p.out, p.B, p.T, p.H, p.Dv);
  if (narrow && !tma) return MXB_ERR_UNSUPPORTED;
  if (tma) {
    if (MXB_ALLOW_SMEM(kPrepSmem, gdn_tc_prep_kernel<true>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_tc_prep_kernel", st,
               (launch_kernel(gdn_tc_prep_kernel<true>, dim3(p.n, p.B * p.H), 128, kPrepSmem, st, p, maps)));
  } else {
    if (MXB_ALLOW_SMEM(kPrepSmem, gdn_tc_prep_kernel<false>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_tc_prep_kernel", st,
               (launch_kernel(gdn_tc_prep_kernel<false>, dim3(p.n, p.B * p.H), 128, kPrepSmem, st, p, maps)));
  }
  mxb_status s = check_launch("gdn_tc_prep_kernel");
  if (s != MXB_OK) return s;
  auto state = [&](auto tma_v, auto nv) {
    constexpr bool TMA = decltype(tma_v)::value;
    constexpr int NV = decltype(nv)::value;
    if (MXB_ALLOW_SMEM(kStateFwdSmem<NV>, gdn_tc_state_fwd_kernel<TMA, NV>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_tc_state_fwd_kernel", st,
               (launch_kernel(gdn_tc_state_fwd_kernel<TMA, NV>, dim3(p.B * p.H, (p.Dv + NV - 1) / NV), kStateThreads<NV>, kStateFwdSmem<NV>, st, p, maps)));
    return MXB_OK;
  };
  if (tma && chain_columns(p, p.save)) return chain_fwd(p, maps, chain_columns(p, p.save), st);
  if (!tma) s = state(std::false_type{}, std::integral_constant<int, KD>{});
  else if (tc_split_columns(p)) s = state(std::true_type{}, std::integral_constant<int, 64>{});
  else s = state(std::true_type{}, std::integral_constant<int, KD>{});
  if (s != MXB_OK) return s;
  return check_launch("gdn_tc_state_fwd_kernel");
}

mxb_status gdn_tc_fwd(const mxb_gdn_desc* d, const void* q, const void* k, const void* v, const float* beta,
                      const float* gate, const float* h0, void* out, float* out32, float* hT, void* ws, cudaStream_t st) {
  TcP p = make_tc(d);
  p.out32 = out32;
  p.q = static_cast<const bf16*>(q); p.k = static_cast<const bf16*>(k); p.v = static_cast<const bf16*>(v);
  p.beta = beta; p.gate = gate; p.h0 = h0; p.out = static_cast<bf16*>(out); p.hT = hT;
  p.save = (d->flags & MXB_GDN_SAVE_FOR_BWD) ? 1 : 0;
  p.no_tma = (d->flags & MXB_GDN_NO_TMA) ? 1 : 0;
  carve_tc(p, ws, p.save != 0);
  return tc_run_fwd(p, st);
}

mxb_status gdn_tc_bwd(const mxb_gdn_desc* d, const void* q, const void* k, const void* v, const float* beta,
                      const float* gate, const float* h0, const void* dO, const float* dhT, void* dq, void* dk,
                      void* dv, float* dq32, float* dk32, float* dv32, float* dbeta, float* dgate, float* dh0, void* ws,
                      cudaStream_t st) {
  if (d->flags & MXB_GDN_BWD_FP32_KERNELS) {  // what a forward saved is in these kernels' layout: the others recompute
    mxb_gdn_desc own = *d;
    own.flags &= ~MXB_GDN_BWD_USE_SAVED;
    return gdn_simt_bwd(&own, q, k, v, beta, gate, h0, dO, dhT, dq, dk, dv, dbeta, dgate, dh0, ws, st);
  }
  TcP p = make_tc(d);
  p.q = static_cast<const bf16*>(q); p.k = static_cast<const bf16*>(k); p.v = static_cast<const bf16*>(v);
  p.beta = beta; p.gate = gate; p.h0 = h0;
  p.dO = static_cast<const bf16*>(dO); p.dhT_in = dhT;
  p.dq = static_cast<bf16*>(dq); p.dk = static_cast<bf16*>(dk); p.dv = static_cast<bf16*>(dv);
  p.dq32 = dq32; p.dk32 = dk32; p.dv32 = dv32;
  p.dbeta = dbeta; p.dgate = dgate; p.dh0 = dh0;
  p.no_tma = (d->flags & MXB_GDN_NO_TMA) ? 1 : 0;
  carve_tc(p, ws, true);
  return tc_run_bwd(p, !(d->flags & MXB_GDN_BWD_USE_SAVED), st);
}

}  // namespace mxb
