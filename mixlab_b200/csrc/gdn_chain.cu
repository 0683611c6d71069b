// Gated delta rule, tensor-core path: the sequential passes where the (batch, head) pairs leave SMs idle.
//
// What counts there is the time from one chunk's state to the next one's.  With tcgen05.mma a link of that chain is two
// products that each cost an issue, a commit, an mbarrier wait and a read of tensor memory (0.45 us from issue to result,
// 1.9 us a chunk with everything around them).  These kernels take mma.sync instead: a product of 16 columns of the state
// takes 0.07 us on four warps and its operands and results are registers.  The rate of mma.sync (a quarter of tcgen05's)
// is no limit here: the columns of the state are independent, so NV of them go to a CTA and the slabs of a head run on
// SMs of their own.
//
// Everything is held transposed, columns of the state as rows of the products, so that an accumulator fragment packed to
// bf16 is the operand fragment of the next product:
//   forward   v_new^T = u^T - S^T w^T              S^T <- E(gam_last) S^T + v_new^T (r k)
//             out^T   = E(gam) (S^T q^T) + v_new^T P^T
//   backward  dv_new^T = r (dS^T k^T) + dO^T P     dS^T <- E(gam_last) dS^T + dO^T (d q) - dv_new^T w
// The mathematics, the workspace tiles, the roundings and the order of every sum are those of gdn_tc.cu, gdn_tc_bwd.cu and
// gdn_tc64.cu, and mma.sync adds the 16 products of a step as tcgen05.mma does: finite results are equal bit for bit, so a
// sequence gives the same bits alone and in a batch that takes the other kernels.  An infinity or NaN spreads differently: the
// products with the zero half of P are skipped here and made there, so there it reaches all rows of its chunk (0 x NaN), here
// the rows that use it and those of its block of 16.
//
// Twelve warps.  Chain warps 0-3, one per scheduler: a quarter of the chunk's rows in the first product, a quarter of the
// state's rows (kept in registers, fp32) in the second; between the two they exchange v_new and S through shared memory as
// the byte images that the other kernels read.  Warps 4-7 make what is not on the chain, a quarter of the rows each: the
// output forward, dO^T P and dO^T (d q) backward.  Warps 8-10 issue the copies of one ring of operand tiles each, warp 11
// hands the images of S and v_new (dS, -dv_new) to the copy engine.  Every hand-over between these groups is an mbarrier
// with a bounded wait; a warp whose wait has run out stops waiting and working but goes through its loop.
//
// A chunk takes 1750 cycles at 16 heads of 128, 24 chunks, 16 columns (tcgen05: 3800): two products 650 + 260, their
// hand-overs 300, and the rest waits for operands: 56 KB a chunk and CTA from L2, which every CTA of a head reads for itself,
// and the 170 KB that go through shared memory.  Scaling k in shared memory (four warps of their own) took 100 cycles more.
#include <cuda.h>

#include <cstring>

#include "gdn_tc.cuh"
#include "mma_sync.cuh"

namespace mxb {
namespace chain {
constexpr int kThreads = 384;

using tc::mbar_arrive;
using ms::ldsm;
using ms::ldsm_t;
using ms::mma;
using ms::stsm_t;
// Two packed bf16 times two floats, rounded back.
__device__ __forceinline__ uint32_t scale2(uint32_t v, float2 s) {
  float a, b;
  tc::unpack_bf16(v, a, b);
  return tc::pack_bf16(a * s.x, b * s.y);
}
// The four chain warps among themselves (they never wait for one another anywhere else, so this needs no limit).
__device__ __forceinline__ void chain_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Tiles.  W: width of the state's rows and of q, k, w (64 or 128 columns), NV: columns of the state per CTA.
//   token tiles (q, k, w): [64][W], slabs of 64 columns in the 128-byte swizzle          -> tc::sw128_unit
//   slabs of the column tiles (u, v_new: 64 rows; S: W rows): the piece of the workspace image that holds these columns,
//   column-blocked for W = 128, groups of eight rows for W = 64                          -> loc
template <int W, int NV>
__device__ __forceinline__ uint32_t loc(int r, int c8, int rows) {
  return W == 128 ? (uint32_t)(c8 * rows + r) * 16u : (uint32_t)(r >> 3) * (NV * 16u) + (uint32_t)c8 * 128u + (uint32_t)(r & 7) * 16u;
}
// The image of `rows` rows in the workspace, this CTA's columns of it: one contiguous piece, or one per eight rows.
template <int W, int NV, typename F>
__device__ __forceinline__ void pieces(bf16* image, int col0, int rows, uint32_t smem, F copy) {
  if (W == 128) {
    copy(image + (size_t)rows * col0, smem, (uint32_t)(rows * NV * 2));
  } else {
    for (int g = 0; g < rows / 8; ++g) copy(image + g * 512 + col0 * 8, smem + g * (NV * 16), (uint32_t)(NV * 16));
  }
}
// The tile of P: [i][m] in 8x8 blocks for W = 128, swizzled for W = 64 (where the forward pass reads P^T, [m][i]).
template <int W>
__device__ __forceinline__ uint32_t p_unit(int r, int c8) {
  return W == 128 ? (uint32_t)(r >> 3) * 1024u + (uint32_t)c8 * 128u + (uint32_t)(r & 7) * 16u
                  : (uint32_t)r * 128u + (uint32_t)((c8 ^ (r & 7)) << 4);
}
// Addresses of this lane's row for fragments of a [rows][cols] tile with offsets unit(row, c8):
//   operand B, contraction along the columns (two groups of eight rows n)
template <typename U>
__device__ __forceinline__ uint32_t b_nat(U unit, int n0, int ks, int lane) {
  return unit(n0 + ((lane >> 4) << 3) + (lane & 7), 2 * ks + ((lane >> 3) & 1));
}
//   operand B, contraction along the rows (two groups of eight columns n)
template <typename U>
__device__ __forceinline__ uint32_t b_trn(U unit, int n8, int ks, int lane) {
  return unit(16 * ks + (lane & 15), n8 + (lane >> 4));
}
//   operand A or a result, transposed: 16 columns of the tile as rows, 16 of its rows as columns
template <typename U>
__device__ __forceinline__ uint32_t a_trn(U unit, int c16, int r0, int lane) {
  return unit(r0 + ((lane >> 4) << 3) + (lane & 7), 2 * c16 + ((lane >> 3) & 1));
}

template <int W, int NV, int NS, int NB>
struct Layout {
  static constexpr int kRow = W * 128;     // bytes of a token tile
  static constexpr int kU = NV * 128;      // of a slab of u, v_new, dO, out
  static constexpr int kS = W * NV * 2;    // of a slab of the state
  static constexpr int kP = 8192;
  static constexpr int bars = 6 * NS + 3 * NB + 2;
};

// --------------------------------------------------------------------------------------------------------- forward
template <int W, int NV, int NS, int NB>
constexpr int kFwdSmem = NS * (3 * W * 128 + NV * 128 + 8192) + NB * (W * NV * 2 + NV * 128) + NV * 128 + 512 + 8 * Layout<W, NV, NS, NB>::bars + 1024;

template <int W, int NV, int NS, int NB>
__global__ void __launch_bounds__(kThreads, 1) gdn_chain_fwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  using L = Layout<W, NV, NS, NB>;
  constexpr int MT = NV / 16, KS = W / 16, NT = W / 32;  // 16-column blocks; steps of a contraction over W; row groups of S per warp
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Rw = sm;                      // xNS w
  uint8_t* Rk = Rw + NS * L::kRow;       // xNS k
  uint8_t* Rq = Rk + NS * L::kRow;       // xNS q
  uint8_t* Rp = Rq + NS * L::kRow;       // xNS P
  uint8_t* Ru = Rp + NS * L::kP;         // xNS u
  uint8_t* So = Ru + NS * L::kU;         // xNB S at chunk start, bf16
  uint8_t* Vn = So + NB * L::kS;         // xNB v_new
  uint8_t* Ot = Vn + NB * L::kU;             // output rows on their way out (each warp its own)
  float* rr = reinterpret_cast<float*>(Ot + L::kU);           // x2 r of a chunk's rows
  uint64_t* fullA = reinterpret_cast<uint64_t*>(rr + 2 * C);  // w and u landed
  uint64_t* fullK = fullA + NS;
  uint64_t* fullQ = fullK + NS;          // q and P landed
  uint64_t* freeA = fullQ + NS;
  uint64_t* freeK = freeA + NS;
  uint64_t* freeQ = freeK + NS;
  uint64_t* sready = freeQ + NS;        // xNB: S of a chunk complete
  uint64_t* vready = sready + NB;        // xNB: v_new of a chunk complete
  uint64_t* odone = vready + NB;         // xNB: output and store warps no longer read the chunk's S and v_new

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H, col0 = blockIdx.y * NV, n = p.n;
  const size_t ci0 = (size_t)bh * n;
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      tc::mbar_init(fullA + s, 1); tc::mbar_init(fullK + s, 1); tc::mbar_init(fullQ + s, 1);
      tc::mbar_init(freeA + s, 4); tc::mbar_init(freeK + s, 4); tc::mbar_init(freeQ + s, 4);
    }
    for (int s = 0; s < NB; ++s) {
      tc::mbar_init(sready + s, 4); tc::mbar_init(vready + s, 4); tc::mbar_init(odone + s, p.save ? 5 : 4);
    }
    tc::mbar_fence_init();
  }
  __syncthreads();
  bool ok = true;
  auto wait = [&](uint64_t* m, int parity) { if (ok) ok = tc::mbar_wait(m, (uint32_t)parity & 1u); };
  auto arrive = [&](uint64_t* m) {  // of a whole warp
    __syncwarp();
    if (lane == 0) mbar_arrive(m);
  };
  auto tile = [](int r, int c8) { return tc::sw128_unit(r, c8); };
  auto slab64 = [](int r, int c8) { return loc<W, NV>(r, c8, 64); };
  auto slabS = [](int r, int c8) { return loc<W, NV>(r, c8, W); };

  if (warp >= 8) {
    tc::reg_dec<40>();
    if (lane == 0) {
      int issued = 0;  // a CTA outlives the copies it has requested, also when a wait has run out
      auto landed = [&](uint64_t* full) {
        for (int q = max(0, issued - NS); q < issued; ++q) tc::mbar_wait(full + q % NS, (q / NS) & 1);
      };
      if (warp == 8) {
        for (int c = 0; c < n; ++c) {
          const int s = c % NS;
          if (c >= NS) wait(freeA + s, c / NS - 1);
          if (!ok) break;
          ++issued;
          tc::mbar_expect_tx(fullA + s, L::kRow + L::kU);
          tc::bulk_load(tc::smem_u32(Rw + s * L::kRow), p.w + (ci0 + c) * C * W, L::kRow, fullA + s);
          pieces<W, NV>(p.u + (ci0 + c) * C * W, col0, 64, tc::smem_u32(Ru + s * L::kU),
                        [&](bf16* g, uint32_t sa, uint32_t bytes) { tc::bulk_load(sa, g, bytes, fullA + s); });
        }
        landed(fullA);
      } else if (warp == 9) {
        for (int c = 0; c < n; ++c) {
          const int s = c % NS;
          if (c >= NS) wait(freeK + s, c / NS - 1);
          if (!ok) break;
          ++issued;
          tc::mbar_expect_tx(fullK + s, L::kRow);
          for (int sl = 0; sl < W / 64; ++sl)
            tc::tma_load_4d(tc::smem_u32(Rk + s * L::kRow) + sl * 8192, &maps.k, 64 * sl, h, c * C, b, fullK + s);
        }
        landed(fullK);
      } else if (warp == 10) {
        const bf16* P = W == 64 ? p.Pt : p.P;
        for (int c = 0; c < n; ++c) {
          const int s = c % NS;
          if (c >= NS) wait(freeQ + s, c / NS - 1);
          if (!ok) break;
          ++issued;
          tc::mbar_expect_tx(fullQ + s, L::kRow + L::kP);
          for (int sl = 0; sl < W / 64; ++sl)
            tc::tma_load_4d(tc::smem_u32(Rq + s * L::kRow) + sl * 8192, &maps.q, 64 * sl, h, c * C, b, fullQ + s);
          tc::bulk_load(tc::smem_u32(Rp + s * L::kP), P + (ci0 + c) * C * C, L::kP, fullQ + s);
        }
        landed(fullQ);
      } else {  // S0 and v_new, saved for the backward as the byte images of the operand tiles
        auto store = [&](bf16* g, uint32_t sa, uint32_t bytes) { tc::bulk_store(g, sa, bytes); };
        for (int c = 0; p.save && c < n && ok; ++c) {
          const int bf = c % NB;
          wait(sready + bf, c / NB);
          if (ok) pieces<W, NV>(p.hs + (ci0 + c) * W * W, col0, W, tc::smem_u32(So + bf * L::kS), store);
          tc::bulk_commit();
          wait(vready + bf, c / NB);
          if (ok) pieces<W, NV>(p.vn + (ci0 + c) * C * W, col0, 64, tc::smem_u32(Vn + bf * L::kU), store);
          tc::bulk_commit();
          tc::bulk_wait_read<0>();
          mbar_arrive(odone + bf);
        }
      }
      if (!ok) atomicExch(p.status, 2);
    }
    return;
  }

  const int w = warp & 3, r0 = 16 * w;  // this warp's rows of the chunk
  const float* gam = p.gam + ci0 * C;
  if (warp < 4) {
    tc::reg_inc<232>();
    const int k0 = (W / 4) * w;          // this warp's rows of the state
    float S[MT][NT][4];                  // S^T: columns 16 m + lane / 4 (+ 8), rows k0 + 8 t + 2 (lane % 4) (+ 1)
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int j = col0 + 16 * m + (lane >> 2) + 8 * (x >> 1), kk = k0 + 8 * t + 2 * (lane & 3) + (x & 1);
          S[m][t][x] = p.h0 && kk < p.Dk && j < p.Dv ? __ldg(p.h0 + ((size_t)bh * p.Dk + kk) * p.Dv + j) : 0.f;
        }
    auto put_S = [&](int bf) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; t += 2)
          stsm_t(tc::smem_u32(So + bf * L::kS) + a_trn(slabS, m, k0 + 8 * t, lane), tc::pack_bf16(S[m][t][0], S[m][t][1]),
                 tc::pack_bf16(S[m][t][2], S[m][t][3]), tc::pack_bf16(S[m][t + 1][0], S[m][t + 1][1]),
                 tc::pack_bf16(S[m][t + 1][2], S[m][t + 1][3]));
      if (p.save) tc::fence_async_smem();
      arrive(sready + bf);
      chain_sync();
    };
    // r of the chunk ahead: each warp fills in its rows, a chunk before they are read
    float gk = gam[r0 + (lane & 15)], gl = gam[C - 1], Ln = exp_nonpos(gl);
    auto decay = [&](int c) {
      if (lane < 16) rr[(c & 1) * C + r0 + lane] = exp_nonpos(gl - gk);
      Ln = exp_nonpos(gl);
      if (c + 1 < n) {
        gk = gam[(c + 1) * C + r0 + (lane & 15)];
        gl = gam[(c + 1) * C + C - 1];
      }
    };
    decay(0);
    put_S(0);
    for (int c = 0; c < n; ++c) {
      const int s = c % NS, bf = c % NB;
      const float Ld = Ln;
      decay(c + 1);
      wait(fullA + s, c / NS);
      uint32_t bw[KS][4], uu[MT][4];
      const uint32_t sw = tc::smem_u32(Rw + s * L::kRow);
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) ldsm(bw[ks], sw + b_nat(tile, r0, ks, lane));
#pragma unroll
      for (int m = 0; m < MT; ++m) ldsm_t(uu[m], tc::smem_u32(Ru + s * L::kU) + a_trn(slab64, m, r0, lane));
      wait(fullK + s, c / NS);
      uint32_t bk[C / 16][NT / 2][4];  // (r k): scaled while the first product goes through its steps
      const uint32_t sk = tc::smem_u32(Rk + s * L::kRow);
#pragma unroll
      for (int ks = 0; ks < C / 16; ++ks)
#pragma unroll
        for (int t = 0; t < NT / 2; ++t) ldsm_t(bk[ks][t], sk + b_trn(tile, k0 / 8 + 2 * t, ks, lane));
      float acc[MT][2][4] = {};
      const uint32_t sS = tc::smem_u32(So + bf * L::kS);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[KS][4];
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) ldsm_t(a[ks], sS + a_trn(slabS, m, 16 * ks, lane));
        if (m == 0) {
#pragma unroll
          for (int ks = 0; ks < C / 16; ++ks) {
            const float2* r2 = reinterpret_cast<const float2*>(rr + (c & 1) * C + 16 * ks) + (lane & 3);
            const float2 ra = r2[0], rb = r2[4];
#pragma unroll
            for (int t = 0; t < NT / 2; ++t)
#pragma unroll
              for (int x = 0; x < 4; ++x) bk[ks][t][x] = scale2(bk[ks][t][x], x & 1 ? rb : ra);
          }
        }
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          mma(acc[m][0], a[ks], bw[ks][0], bw[ks][1]);
          mma(acc[m][1], a[ks], bw[ks][2], bw[ks][3]);
        }
      }
      arrive(freeA + s);
      arrive(freeK + s);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        float v[2][4];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          tc::unpack_bf16(uu[m][2 * t], v[t][0], v[t][1]);
          tc::unpack_bf16(uu[m][2 * t + 1], v[t][2], v[t][3]);
#pragma unroll
          for (int x = 0; x < 4; ++x) v[t][x] -= acc[m][t][x];
        }
        stsm_t(tc::smem_u32(Vn + bf * L::kU) + a_trn(slab64, m, r0, lane), tc::pack_bf16(v[0][0], v[0][1]),
               tc::pack_bf16(v[0][2], v[0][3]), tc::pack_bf16(v[1][0], v[1][1]), tc::pack_bf16(v[1][2], v[1][3]));
      }
      if (p.save) tc::fence_async_smem();
      arrive(vready + bf);
      chain_sync();
      float up[MT][NT][4] = {};
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[C / 16][4];
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks) ldsm_t(a[ks], tc::smem_u32(Vn + bf * L::kU) + a_trn(slab64, m, 16 * ks, lane));
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks)
#pragma unroll
          for (int t = 0; t < NT / 2; ++t) {
            mma(up[m][2 * t], a[ks], bk[ks][t][0], bk[ks][t][1]);
            mma(up[m][2 * t + 1], a[ks], bk[ks][t][2], bk[ks][t][3]);
          }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int x = 0; x < 4; ++x) S[m][t][x] = fmaf(Ld, S[m][t][x], up[m][t][x]);
      if (c + 1 < n) {
        if (c + 1 >= NB) wait(odone + (c + 1) % NB, (c + 1) / NB - 1);
        put_S((c + 1) % NB);
      }
    }
    if (ok && p.hT) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int j = col0 + 16 * m + (lane >> 2) + 8 * (x >> 1), kk = k0 + 8 * t + 2 * (lane & 3) + (x & 1);
            if (kk < p.Dk && j < p.Dv) p.hT[((size_t)bh * p.Dk + kk) * p.Dv + j] = S[m][t][x];
          }
    }
  } else {
    tc::reg_inc<232>();  // (232 + 232 + 40 registers a lane, of 3 x 168 at launch)
    const int tk = r0 + 2 * (lane & 3);
    float2 g0 = *reinterpret_cast<const float2*>(gam + tk), g1 = *reinterpret_cast<const float2*>(gam + tk + 8);
    for (int c = 0; c < n; ++c) {
      const int s = c % NS, bf = c % NB;
      const float d[4] = {exp_nonpos(g0.x), exp_nonpos(g0.y), exp_nonpos(g1.x), exp_nonpos(g1.y)};
      if (c + 1 < n) {
        const float* gn = gam + (c + 1) * C;
        g0 = *reinterpret_cast<const float2*>(gn + tk);
        g1 = *reinterpret_cast<const float2*>(gn + tk + 8);
      }
      wait(fullQ + s, c / NS);
      uint32_t bq[KS][4];
      const uint32_t sq = tc::smem_u32(Rq + s * L::kRow), sp = tc::smem_u32(Rp + s * L::kP);
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) ldsm(bq[ks], sq + b_nat(tile, r0, ks, lane));
      wait(sready + bf, c / NB);
      float acc[MT][2][4] = {};
      const uint32_t sS = tc::smem_u32(So + bf * L::kS);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[KS][4];
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) ldsm_t(a[ks], sS + a_trn(slabS, m, 16 * ks, lane));
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          mma(acc[m][0], a[ks], bq[ks][0], bq[ks][1]);
          mma(acc[m][1], a[ks], bq[ks][2], bq[ks][3]);
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[m][t][x] *= d[2 * t + (x & 1)];
      wait(vready + bf, c / NB);
      float pv[MT][2][4] = {};
#pragma unroll
      for (int ks = 0; ks < C / 16; ++ks)
        if (ks <= w) {  // P is lower triangular
          uint32_t bp[4];
          if (W == 128) ldsm(bp, sp + b_nat(p_unit<W>, r0, ks, lane));
          else ldsm_t(bp, sp + b_trn(p_unit<W>, r0 / 8, ks, lane));
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            uint32_t a[4];
            ldsm_t(a, tc::smem_u32(Vn + bf * L::kU) + a_trn(slab64, m, 16 * ks, lane));
            mma(pv[m][0], a, bp[0], bp[1]);
            mma(pv[m][1], a, bp[2], bp[3]);
          }
        }
      arrive(odone + bf);
      arrive(freeQ + s);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[m][t][x] += pv[m][t][x];
#pragma unroll
      for (int m = 0; m < MT; ++m)
        stsm_t(tc::smem_u32(Ot) + a_trn(slab64, m, r0, lane), tc::pack_bf16(acc[m][0][0], acc[m][0][1]),
               tc::pack_bf16(acc[m][0][2], acc[m][0][3]), tc::pack_bf16(acc[m][1][0], acc[m][1][1]),
               tc::pack_bf16(acc[m][1][2], acc[m][1][3]));
      __syncwarp();
      if (ok) {
#pragma unroll
        for (int u = lane; u < 16 * (NV / 8); u += 32) {
          const int i = r0 + u / (NV / 8), c8 = u % (NV / 8);
          const uint4 val = *reinterpret_cast<const uint4*>(Ot + slab64(i, c8));
          if (c * C + i < p.T && col0 + 8 * c8 < p.Dv) {
            const size_t o = ((size_t)(b * p.T + c * C + i) * p.H + h) * p.Dv + col0 + 8 * c8;
            if (p.out32) put_wide(p.out32 + o, val);
            else *reinterpret_cast<uint4*>(p.out + o) = val;
          }
        }
      }
      __syncwarp();
    }
  }
  if (!ok && lane == 0) atomicExch(p.status, 2);
}

// -------------------------------------------------------------------------------------------------------- backward
template <int W, int NV, int NS, int NB>
constexpr int kBwdSmem = NS * (3 * W * 128 + NV * 128 + 8192) + NB * (W * NV * 2 + NV * 128) +
                         (64 * NV * 4 + W * NV * 4) + 8 * Layout<W, NV, NS, NB>::bars + 1024;

template <int W, int NV, int NS, int NB>
__global__ void __launch_bounds__(kThreads, 1) gdn_chain_bwd_kernel(TcP p, const __grid_constant__ RowMaps maps) {
  begin_dependent();
  using L = Layout<W, NV, NS, NB>;
  constexpr int MT = NV / 16, KS = W / 16, NT = W / 32;
  constexpr int kX = 64 * NV * 4, kY = W * NV * 4;  // dO^T P and dO^T (d q), fp32 fragments
  extern __shared__ uint8_t raw[];
  uint8_t* sm = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
  uint8_t* Rk = sm;                      // xNS k
  uint8_t* Rw = Rk + NS * L::kRow;       // xNS w
  uint8_t* Rq = Rw + NS * L::kRow;       // xNS q
  uint8_t* Rp = Rq + NS * L::kRow;       // xNS P
  uint8_t* Rd = Rp + NS * L::kP;         // xNS dO, these columns (rows of NV columns, swizzled over their width)
  uint8_t* So = Rd + NS * L::kU;         // xNB dS at chunk end, bf16
  uint8_t* Vn = So + NB * L::kS;         // xNB -dv_new
  uint8_t* X = Vn + NB * L::kU;          // the other warps compute a step ahead and hold their results in registers
  uint8_t* Y = X + kX;
  uint64_t* fullK = reinterpret_cast<uint64_t*>(Y + kY);
  uint64_t* fullW = fullK + NS;
  uint64_t* fullQ = fullW + NS;          // q, P and dO landed
  uint64_t* freeK = fullQ + NS;
  uint64_t* freeW = freeK + NS;
  uint64_t* freeQ = freeW + NS;
  uint64_t* sready = freeQ + NS;        // xNB: dS of a chunk complete
  uint64_t* vready = sready + NB;        // xNB: -dv_new of a chunk complete
  uint64_t* sdone = vready + NB;         // xNB: the images of dS and -dv_new have left
  uint64_t* xready = sdone + NB;         // X and Y of a chunk complete
  uint64_t* xdone = xready + 1;          // and taken

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H, col0 = blockIdx.y * NV, n = p.n;
  const size_t ci0 = (size_t)bh * n;
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      tc::mbar_init(fullK + s, 1); tc::mbar_init(fullW + s, 1); tc::mbar_init(fullQ + s, 1);
      tc::mbar_init(freeK + s, 4); tc::mbar_init(freeW + s, 4); tc::mbar_init(freeQ + s, 4);
    }
    for (int s = 0; s < NB; ++s) {
      tc::mbar_init(sready + s, 4); tc::mbar_init(vready + s, 4); tc::mbar_init(sdone + s, 1);
    }
    tc::mbar_init(xready, 4);
    tc::mbar_init(xdone, 4);
    tc::mbar_fence_init();
  }
  __syncthreads();
  bool ok = true;
  auto wait = [&](uint64_t* m, int parity) { if (ok) ok = tc::mbar_wait(m, (uint32_t)parity & 1u); };
  auto arrive = [&](uint64_t* m) {
    __syncwarp();
    if (lane == 0) mbar_arrive(m);
  };
  auto tile = [](int r, int c8) { return tc::sw128_unit(r, c8); };
  auto slab64 = [](int r, int c8) { return loc<W, NV>(r, c8, 64); };
  auto slabS = [](int r, int c8) { return loc<W, NV>(r, c8, W); };
  // dO: rows of 2 NV bytes; the copy engine swaps the 16-byte units of a row within its 32, 64 or 128 bytes
  auto dOu = [](int r, int c8) {
    const uint32_t x = (uint32_t)r * (2 * NV) + (uint32_t)c8 * 16u;
    return x ^ (((x >> 7) & (NV / 8 - 1)) << 4);
  };
  // step e of the pass works on chunk n - 1 - e

  if (warp >= 8) {
    tc::reg_dec<40>();
    if (lane == 0) {
      int issued = 0;
      auto landed = [&](uint64_t* full) {
        for (int q = max(0, issued - NS); q < issued; ++q) tc::mbar_wait(full + q % NS, (q / NS) & 1);
      };
      if (warp == 8) {
        for (int e = 0; e < n; ++e) {
          const int s = e % NS, c = n - 1 - e;
          if (e >= NS) wait(freeK + s, e / NS - 1);
          if (!ok) break;
          ++issued;
          tc::mbar_expect_tx(fullK + s, L::kRow);
          for (int sl = 0; sl < W / 64; ++sl)
            tc::tma_load_4d(tc::smem_u32(Rk + s * L::kRow) + sl * 8192, &maps.k, 64 * sl, h, c * C, b, fullK + s);
        }
        landed(fullK);
      } else if (warp == 9) {
        for (int e = 0; e < n; ++e) {
          const int s = e % NS, c = n - 1 - e;
          if (e >= NS) wait(freeW + s, e / NS - 1);
          if (!ok) break;
          ++issued;
          tc::mbar_expect_tx(fullW + s, L::kRow);
          tc::bulk_load(tc::smem_u32(Rw + s * L::kRow), p.w + (ci0 + c) * C * W, L::kRow, fullW + s);
        }
        landed(fullW);
      } else if (warp == 10) {
        for (int e = 0; e < n; ++e) {
          const int s = e % NS, c = n - 1 - e;
          if (e >= NS) wait(freeQ + s, e / NS - 1);
          if (!ok) break;
          ++issued;
          tc::mbar_expect_tx(fullQ + s, L::kRow + L::kP + L::kU);
          for (int sl = 0; sl < W / 64; ++sl)
            tc::tma_load_4d(tc::smem_u32(Rq + s * L::kRow) + sl * 8192, &maps.q, 64 * sl, h, c * C, b, fullQ + s);
          tc::bulk_load(tc::smem_u32(Rp + s * L::kP), p.P + (ci0 + c) * C * C, L::kP, fullQ + s);
          tc::tma_load_4d(tc::smem_u32(Rd + s * L::kU), &maps.dO, col0, h, c * C, b, fullQ + s);
        }
        landed(fullQ);
      } else {  // dS at chunk end and -dv_new, for the chunk kernel
        auto store = [&](bf16* g, uint32_t sa, uint32_t bytes) { tc::bulk_store(g, sa, bytes); };
        for (int e = 0; e < n && ok; ++e) {
          const int bf = e % NB, c = n - 1 - e;
          wait(sready + bf, e / NB);
          if (ok) pieces<W, NV>(p.dhs + (ci0 + c) * W * W, col0, W, tc::smem_u32(So + bf * L::kS), store);
          tc::bulk_commit();
          wait(vready + bf, e / NB);
          if (ok) pieces<W, NV>(p.dvn + (ci0 + c) * C * W, col0, 64, tc::smem_u32(Vn + bf * L::kU), store);
          tc::bulk_commit();
          tc::bulk_wait_read<0>();
          mbar_arrive(sdone + bf);
        }
      }
      if (!ok) atomicExch(p.status, 3);
    }
    return;
  }

  const int w = warp & 3, r0 = 16 * w, k0 = (W / 4) * w;
  const float* gam = p.gam + ci0 * C;
  if (warp < 4) {
    tc::reg_inc<232>();
    float S[MT][NT][4];  // dS^T
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int j = col0 + 16 * m + (lane >> 2) + 8 * (x >> 1), kk = k0 + 8 * t + 2 * (lane & 3) + (x & 1);
          S[m][t][x] = p.dhT_in && kk < p.Dk && j < p.Dv ? __ldg(p.dhT_in + ((size_t)bh * p.Dk + kk) * p.Dv + j) : 0.f;
        }
    auto put_S = [&](int bf) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; t += 2)
          stsm_t(tc::smem_u32(So + bf * L::kS) + a_trn(slabS, m, k0 + 8 * t, lane), tc::pack_bf16(S[m][t][0], S[m][t][1]),
                 tc::pack_bf16(S[m][t][2], S[m][t][3]), tc::pack_bf16(S[m][t + 1][0], S[m][t + 1][1]),
                 tc::pack_bf16(S[m][t + 1][2], S[m][t + 1][3]));
      tc::fence_async_smem();
      arrive(sready + bf);
      chain_sync();
    };
    put_S(0);
    const int tk = r0 + 2 * (lane & 3);
    const float* gn = gam + (size_t)(n - 1) * C;
    float2 g0 = *reinterpret_cast<const float2*>(gn + tk), g1 = *reinterpret_cast<const float2*>(gn + tk + 8);
    float gl = gn[C - 1];
    for (int e = 0; e < n; ++e) {
      const int s = e % NS, bf = e % NB;
      const float r[4] = {exp_nonpos(gl - g0.x), exp_nonpos(gl - g0.y), exp_nonpos(gl - g1.x), exp_nonpos(gl - g1.y)};
      const float Ld = exp_nonpos(gl);
      if (e + 1 < n) {
        gn -= C;
        g0 = *reinterpret_cast<const float2*>(gn + tk);
        g1 = *reinterpret_cast<const float2*>(gn + tk + 8);
        gl = gn[C - 1];
      }
      wait(fullK + s, e / NS);
      uint32_t bk[KS][4];
      const uint32_t sk = tc::smem_u32(Rk + s * L::kRow);
#pragma unroll
      for (int ks = 0; ks < KS; ++ks) ldsm(bk[ks], sk + b_nat(tile, r0, ks, lane));
      wait(xready, e);
      float acc[MT][2][4] = {};
      const uint32_t sS = tc::smem_u32(So + bf * L::kS);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[KS][4];
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) ldsm_t(a[ks], sS + a_trn(slabS, m, 16 * ks, lane));
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          mma(acc[m][0], a[ks], bk[ks][0], bk[ks][1]);
          mma(acc[m][1], a[ks], bk[ks][2], bk[ks][3]);
        }
      }
      arrive(freeK + s);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        float v[2][4];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const float4 x4 = reinterpret_cast<const float4*>(X)[((w * MT + m) * 2 + t) * 32 + lane];
          const float xv[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
          for (int x = 0; x < 4; ++x) v[t][x] = -fmaf(r[2 * t + (x & 1)], acc[m][t][x], xv[x]);
        }
        stsm_t(tc::smem_u32(Vn + bf * L::kU) + a_trn(slab64, m, r0, lane), tc::pack_bf16(v[0][0], v[0][1]),
               tc::pack_bf16(v[0][2], v[0][3]), tc::pack_bf16(v[1][0], v[1][1]), tc::pack_bf16(v[1][2], v[1][3]));
      }
      tc::fence_async_smem();
      arrive(vready + bf);
      chain_sync();
      float up[MT][NT][4];  // (d q)^T dO so far
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const float4 y = reinterpret_cast<const float4*>(Y)[((w * MT + m) * NT + t) * 32 + lane];
          up[m][t][0] = y.x; up[m][t][1] = y.y; up[m][t][2] = y.z; up[m][t][3] = y.w;
        }
      arrive(xdone);
      wait(fullW + s, e / NS);
      uint32_t bw[C / 16][NT / 2][4];
      const uint32_t sw = tc::smem_u32(Rw + s * L::kRow);
#pragma unroll
      for (int ks = 0; ks < C / 16; ++ks)
#pragma unroll
        for (int t = 0; t < NT / 2; ++t) ldsm_t(bw[ks][t], sw + b_trn(tile, k0 / 8 + 2 * t, ks, lane));
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[C / 16][4];
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks) ldsm_t(a[ks], tc::smem_u32(Vn + bf * L::kU) + a_trn(slab64, m, 16 * ks, lane));
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks)
#pragma unroll
          for (int t = 0; t < NT / 2; ++t) {
            mma(up[m][2 * t], a[ks], bw[ks][t][0], bw[ks][t][1]);
            mma(up[m][2 * t + 1], a[ks], bw[ks][t][2], bw[ks][t][3]);
          }
      }
      arrive(freeW + s);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int x = 0; x < 4; ++x) S[m][t][x] = fmaf(Ld, S[m][t][x], up[m][t][x]);
      if (e + 1 < n) {
        if (e + 1 >= NB) wait(sdone + (e + 1) % NB, (e + 1) / NB - 1);
        put_S((e + 1) % NB);
      }
    }
    if (ok && p.dh0) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int j = col0 + 16 * m + (lane >> 2) + 8 * (x >> 1), kk = k0 + 8 * t + 2 * (lane & 3) + (x & 1);
            if (kk < p.Dk && j < p.Dv) p.dh0[((size_t)bh * p.Dk + kk) * p.Dv + j] = S[m][t][x];
          }
    }
  } else {
    tc::reg_inc<232>();
    const float* gn = gam + (size_t)(n - 1) * C + 2 * (lane & 3);
    for (int e = 0; e < n; ++e, gn -= C) {
      const int s = e % NS;
      float2 d[8];  // E(gam) of rows 8 x + 2 (lane % 4) (+ 1)
#pragma unroll
      for (int x = 0; x < 8; ++x) d[x] = *reinterpret_cast<const float2*>(gn + 8 * x);
#pragma unroll
      for (int x = 0; x < 8; ++x) d[x] = make_float2(exp_nonpos(d[x].x), exp_nonpos(d[x].y));
      wait(fullQ + s, e / NS);
      const uint32_t sq = tc::smem_u32(Rq + s * L::kRow), sp = tc::smem_u32(Rp + s * L::kP), sd = tc::smem_u32(Rd + s * L::kU);
      float ax[MT][2][4] = {}, ay[MT][NT][4] = {};
      uint32_t bp[C / 16][4], bq[C / 16][NT / 2][4];
#pragma unroll
      for (int ks = 0; ks < C / 16; ++ks) {
        if (ks >= w) ldsm_t(bp[ks], sp + b_trn(p_unit<W>, r0 / 8, ks, lane));  // P is lower triangular
#pragma unroll
        for (int t = 0; t < NT / 2; ++t) {
          ldsm_t(bq[ks][t], sq + b_trn(tile, k0 / 8 + 2 * t, ks, lane));
#pragma unroll
          for (int x = 0; x < 4; ++x) bq[ks][t][x] = scale2(bq[ks][t][x], d[2 * ks + (x & 1)]);
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[C / 16][4];
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks) ldsm_t(a[ks], sd + a_trn(dOu, m, 16 * ks, lane));
#pragma unroll
        for (int ks = 0; ks < C / 16; ++ks) {
          if (ks >= w) {
            mma(ax[m][0], a[ks], bp[ks][0], bp[ks][1]);
            mma(ax[m][1], a[ks], bp[ks][2], bp[ks][3]);
          }
#pragma unroll
          for (int t = 0; t < NT / 2; ++t) {
            mma(ay[m][2 * t], a[ks], bq[ks][t][0], bq[ks][t][1]);
            mma(ay[m][2 * t + 1], a[ks], bq[ks][t][2], bq[ks][t][3]);
          }
        }
      }
      arrive(freeQ + s);
      if (e > 0) wait(xdone, e - 1);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
#pragma unroll
        for (int t = 0; t < 2; ++t)
          reinterpret_cast<float4*>(X)[((w * MT + m) * 2 + t) * 32 + lane] = make_float4(ax[m][t][0], ax[m][t][1], ax[m][t][2], ax[m][t][3]);
#pragma unroll
        for (int t = 0; t < NT; ++t)
          reinterpret_cast<float4*>(Y)[((w * MT + m) * NT + t) * 32 + lane] = make_float4(ay[m][t][0], ay[m][t][1], ay[m][t][2], ay[m][t][3]);
      }
      arrive(xready);
    }
  }
  if (!ok && lane == 0) atomicExch(p.status, 3);
}
}  // namespace chain

// Columns of the state per CTA of these kernels, 0 where the tcgen05 passes are the better ones: 16 or 32, the fewer that
// keeps every CTA on an SM of its own.  Both passes of 16 heads, 2048 steps, us, tcgen05 against 16 and 32 columns here:
//   128 wide   1 sequence 62 + 58, 43 + 43, 54 + 51     2 sequences 63 + 60, -, 54 + 52
//   64 wide    1 sequence 64 + 56, 32 + 33, 40 + 39     4 sequences 64 + 56, -, 42 + 42
// With 64 columns (twice the sequences) the rate of mma.sync tells: 93 + 80 against 63 + 60, and 66 + 58 against 65 + 57.
int chain_columns(const TcP& p, bool whole) {
  const int W = p.Dk == 64 && p.Dv == 64 ? 64 : 128, width = whole ? W : p.Dv;
  for (int nv = 16; nv <= 32; nv *= 2)
    if (p.B * p.H * ((width + nv - 1) / nv) <= 148) return nv;
  return 0;
}
template <int W, int NV, int NS, int NB, bool BWD>
static mxb_status chain_launch(const TcP& p, const RowMaps& maps, int width, cudaStream_t st) {
  const dim3 grid(p.B * p.H, (width + NV - 1) / NV);
  if constexpr (BWD) {
    constexpr int smem = chain::kBwdSmem<W, NV, NS, NB>;
    static_assert(smem <= 227 * 1024, "");
    if (MXB_ALLOW_SMEM(smem, chain::gdn_chain_bwd_kernel<W, NV, NS, NB>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_chain_bwd_kernel", st, (launch_kernel(chain::gdn_chain_bwd_kernel<W, NV, NS, NB>, grid, chain::kThreads, smem, st, p, maps)));
  } else {
    constexpr int smem = chain::kFwdSmem<W, NV, NS, NB>;
    static_assert(smem <= 227 * 1024, "");
    if (MXB_ALLOW_SMEM(smem, chain::gdn_chain_fwd_kernel<W, NV, NS, NB>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_chain_fwd_kernel", st, (launch_kernel(chain::gdn_chain_fwd_kernel<W, NV, NS, NB>, grid, chain::kThreads, smem, st, p, maps)));
  }
  return check_launch("gdn_chain kernels");
}
mxb_status chain_fwd(const TcP& p, const RowMaps& maps, int nv, cudaStream_t st) {
  const bool w64 = p.Dk == 64 && p.Dv == 64;
  const int width = p.save ? (w64 ? 64 : 128) : p.Dv;
  if (w64) return nv == 16 ? chain_launch<64, 16, 4, 4, false>(p, maps, width, st) : chain_launch<64, 32, 4, 4, false>(p, maps, width, st);
  return nv == 16 ? chain_launch<128, 16, 3, 4, false>(p, maps, width, st) : chain_launch<128, 32, 3, 2, false>(p, maps, width, st);
}
mxb_status chain_bwd(const TcP& p, const RowMaps& maps, int nv, cudaStream_t st) {
  RowMaps m = maps;
  if (!make_tma_map_cols(&m.dO, p.dO, p.B, p.T, p.H, p.Dv, nv)) return MXB_ERR_UNSUPPORTED;
  const bool w64 = p.Dk == 64 && p.Dv == 64;
  const int width = w64 ? 64 : 128;
  if (w64) return nv == 16 ? chain_launch<64, 16, 4, 3, true>(p, m, width, st) : chain_launch<64, 32, 4, 3, true>(p, m, width, st);
  return nv == 16 ? chain_launch<128, 16, 3, 3, true>(p, m, width, st) : chain_launch<128, 32, 2, 2, true>(p, m, width, st);
}
}  // namespace mxb
