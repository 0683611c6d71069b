// Shared declarations of the tensor-core gated-delta kernels (forward: gdn_tc.cu,
// backward: gdn_tc_bwd.cu).
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "umma_tiles.cuh"

namespace mxb {

// [B,T,H,D] bf16 -> tensor map over (D, H, T, B) with 64 x 64 boxes and 128-byte swizzle; false if it cannot be made.
bool make_tma_map_bthd(CUtensorMap* m, const void* base, int B, int T, int H, int D);
// The same with boxes of 16 or 32 columns, swizzled over their own width.
bool make_tma_map_cols(CUtensorMap* m, const void* base, int B, int T, int H, int D, int cols);

namespace tcg {
constexpr int C = 64;     // chunk
constexpr int KD = 128;   // Dk = Dv
constexpr int LDA = 68;   // fp32 row pitch of the 64x64 solve matrix (16-byte aligned rows)
using bf16 = __nv_bfloat16;
using tc::pack8;
using tc::unpack8;

struct TcP {
  int B, T, H, n, gate_is_log, save, no_tma;
  int Dk, Dv;    // true widths of q,k and of v,out (multiples of 8 up to KD).  The tiles are always KD wide: the copy
                 // engine zero-fills the columns a narrower tensor does not have and clips them on the way out, so
                 // only the kernels' direct accesses to the fp32 states index with these
  const bf16 *q, *k, *v;
  const float *beta, *gate, *h0;
  bf16* out;
  float* hT;
  const bf16* dO;
  const float* dhT_in;
  bf16 *dq, *dk, *dv;
  // float32 tensors on these kernels: the results go there, rounded to bf16 all the same, and the bf16 tensors above are scratch
  float *out32, *dq32, *dk32, *dv32;
  float *dbeta, *dgate, *dh0;
  int* status;   // device word: nonzero when a bounded wait gave up
  // workspace, indexed by ci = (b*H+h)*n + chunk
  float* gam;    // [C]
  bf16* Tm;      // [C][C]
  bf16* w;       // [C][KD]
  bf16* u;       // [C][KD]
  bf16* P;       // [C][C]
  bf16* Pt;      // [C][C]    P^T (64-wide kernels only)
  // Everything below is stored as the byte image of the blocked shared-memory operand tile it is read into.
  bf16* hs;      // [KD][KD]  state at chunk start   (backward only)
  bf16* vn;      // [C][KD]
  bf16* dhs;     // [KD][KD]  dS at chunk end
  bf16* dvn;     // [C][KD]   -dv_new (the sign the state pass needs as an operand)
};

// Tensor maps of the token-indexed operands: [B,T,H,128] bf16 viewed as (D, H, T, B), boxes of 64 columns x
// 64 time steps with 128-byte swizzle; rows past the end of the sequence are zero-filled by the copy engine.
// o, dq, dk, dv: results written back by tiled stores (rows past the end of the sequence are clipped).
struct alignas(64) RowMaps {
  CUtensorMap k, q, v, dO, o, dq, dk, dv;
};

__device__ __forceinline__ float log_gate_tc(float g, int gate_is_log) {
  return gate_is_log ? fmaxf(g, kLogGateFloor) : __logf(fmaxf(g, kGateFloor));
}
__device__ __forceinline__ void sts16(uint8_t* base, uint32_t off, uint4 v) {
  *reinterpret_cast<uint4*>(base + off) = v;
}
// Staging-loop index u -> (row, 16-byte unit) of a tile with 16 (or 8) units per row, ordered so that the
// eight lanes of one shared-memory write phase fill one contiguous 128-byte row group of the blocked layout
// (no bank conflicts) while each row is still read from global memory in 64-byte pieces.
__device__ __forceinline__ int urow16(int u) { return ((u >> 7) << 3) | (u & 7); }
__device__ __forceinline__ int ucol16(int u) { return (u >> 3) & 15; }
__device__ __forceinline__ int urow8(int u) { return ((u >> 6) << 3) | (u & 7); }
__device__ __forceinline__ int ucol8(int u) { return (u >> 3) & 7; }
// Eight bf16 as floats (a bf16 is the upper half of the float with the same value).
__device__ __forceinline__ void put_wide(float* dst, uint4 v) {
  reinterpret_cast<float4*>(dst)[0] = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u),
                                                  __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
  reinterpret_cast<float4*>(dst)[1] = make_float4(__uint_as_float(v.z << 16), __uint_as_float(v.z & 0xffff0000u),
                                                  __uint_as_float(v.w << 16), __uint_as_float(v.w & 0xffff0000u));
}
// A finished tile in the layout of a TMA box as rows of a float32 tensor [B,T,H,D], by 256 threads; row0: its first row.
__device__ __forceinline__ void put_wide_tile(float* dst, const uint8_t* tile, size_t row0, int H, int D, int imax) {
  const int w8 = D / 8;
  for (int u = threadIdx.x; u < imax * w8; u += 256) {
    const int i = u / w8, c8 = u % w8;
    put_wide(dst + (row0 + (size_t)i * H) * D + 8 * c8, *reinterpret_cast<const uint4*>(tile + tc::sw128_unit(i, c8)));
  }
}
__device__ __forceinline__ uint4 zero16() { return make_uint4(0u, 0u, 0u, 0u); }

// Loads 32 fp32 accumulator columns [c0, c0+32) of this thread's TMEM lane.
__device__ __forceinline__ void ld_acc32(uint32_t taddr, int warp, int c0, float (&f)[32]) {
  uint32_t r[32];
  tc::tmem_ld_32x32b_x32(taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, r);
  tc::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[i]);
}
// The sequential passes of 128-wide heads take half of the state's columns per CTA where that still puts every CTA on an
// SM of its own: the chain of a chunk is what counts then, not the bytes (forward and backward, us a chunk: 2.55 and 2.4
// with all columns, 1.9 and 1.8 with half of them).  Fewer heads yet: gdn_chain.cu.
inline bool tc_split_columns(const TcP& p) { return p.Dv > 64 && 2 * p.B * p.H <= 148; }

// Threads of a forward state-pass CTA: 256 that hold the state and run the epilogues, and a warp of one issuing thread (on
// a thread with an epilogue of its own, 70 cycles per product made that thread's warp the one all others waited for: 2.4
// -> 1.9 us a chunk with NV = 64, 2.8 -> 2.55 with 128).  With 128 columns per CTA that warp is a warpgroup, so that
// registers can be moved to the others: 8 x 216 + 4 x 40 registers a lane, of 12 x 168 at launch.
template <int NV>
constexpr int kStateThreads = NV == KD ? 384 : 288;

__device__ __forceinline__ void ld_acc16(uint32_t taddr, int warp, int c0, float (&f)[16]) {
  uint32_t r[16];
  tc::tmem_ld_32x32b_x16(taddr + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, r);
  tc::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(r[i]);
}
// Loads 64 fp32 accumulator columns [0, 64) at taddr of this thread's TMEM lane: both loads in flight, one wait.
__device__ __forceinline__ void ld_acc64(uint32_t taddr, int warp, float (&f)[64]) {
  uint32_t r0[32], r1[32];
  const uint32_t base = taddr + ((uint32_t)(32 * (warp & 3)) << 16);
  tc::tmem_ld_32x32b_x32(base, r0);
  tc::tmem_ld_32x32b_x32(base + 32u, r1);
  tc::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    f[i] = __uint_as_float(r0[i]);
    f[32 + i] = __uint_as_float(r1[i]);
  }
}
__device__ __forceinline__ void ld_accN(uint32_t taddr, int warp, float (&f)[64]) { ld_acc64(taddr, warp, f); }
__device__ __forceinline__ void ld_accN(uint32_t taddr, int warp, float (&f)[32]) { ld_acc32(taddr, warp, 0, f); }
__device__ __forceinline__ void ld_accN(uint32_t taddr, int warp, float (&f)[16]) { ld_acc16(taddr, warp, 0, f); }
// T = (I - A)^-1 in fp32, in place over the strictly lower triangular [64][LDA] matrix A; 128 threads, `other(t)` is run
// by threads 64 + t beside the first step.  The four 16 x 16 diagonal blocks by forward substitution (thread = block and
// column, the column in registers), then pairs of blocks are joined twice, T21 = T22 (A21 T11): 16-wide for both halves
// side by side, then 32-wide.  The products take 2 x 2 and 4 x 2 outputs per thread and skip the zero triangle: shared
// memory is what bounds the prep kernels (two 32-step substitutions and one row of 8 outputs per thread took 4.1 k + 2.2 k
// cycles of a CTA's 18 k).  The upper-right blocks are left with A21 T11, nobody reads them.  Ends with a barrier.
template <typename F>
__device__ __forceinline__ void invert_unit_lower(float* Am, bool ok, F other) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  {
    float Tc[16];
    const int r0 = 16 * (tid >> 4), col = tid & 15;
    if (ok && tid < C) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float* arow = Am + (r0 + i) * LDA + r0;
        float s0 = (i == col) ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
        for (int j = 0; j + 1 < i; j += 2) {
          s0 = fmaf(arow[j], Tc[j], s0);
          s1 = fmaf(arow[j + 1], Tc[j + 1], s1);
        }
        if (i & 1) s0 = fmaf(arow[i - 1], Tc[i - 1], s0);
        Tc[i] = (i < col) ? 0.f : s0 + s1;
      }
    } else if (ok) {
      other(tid - C);
    }
    __syncthreads();  // every thread has read its block of A
    if (ok && tid < C) {
#pragma unroll
      for (int i = 0; i < 16; ++i) Am[(r0 + i) * LDA + r0 + col] = Tc[i];
    }
    __syncthreads();
  }
  // out[row0 + rstep r][0, 1] = sum over k in [k0, k1) of a[row0 + rstep r][k] b[k][0, 1]
  auto product = [&](auto rows, const float* a, const float* b, int k0, int k1, int row0, int rstep, float* out) {
    constexpr int R = decltype(rows)::value;
    float x[R][2] = {};
#pragma unroll 2
    for (int k = k0; k < k1; k += 4) {
      float4 av[R];
      float2 bv[4];
#pragma unroll
      for (int r = 0; r < R; ++r) av[r] = *reinterpret_cast<const float4*>(a + (row0 + rstep * r) * LDA + k);
#pragma unroll
      for (int y = 0; y < 4; ++y) bv[y] = *reinterpret_cast<const float2*>(b + (k + y) * LDA);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        x[r][0] = fmaf(av[r].x, bv[0].x, x[r][0]); x[r][1] = fmaf(av[r].x, bv[0].y, x[r][1]);
        x[r][0] = fmaf(av[r].y, bv[1].x, x[r][0]); x[r][1] = fmaf(av[r].y, bv[1].y, x[r][1]);
        x[r][0] = fmaf(av[r].z, bv[2].x, x[r][0]); x[r][1] = fmaf(av[r].z, bv[2].y, x[r][1]);
        x[r][0] = fmaf(av[r].w, bv[3].x, x[r][0]); x[r][1] = fmaf(av[r].w, bv[3].y, x[r][1]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) *reinterpret_cast<float2*>(out + (row0 + rstep * r) * LDA) = make_float2(x[r][0], x[r][1]);
  };
  {  // the two 32 x 32 diagonal blocks: half a CTA each, rows g, g + 8, two columns
    const std::integral_constant<int, 2> two;
    float* M = Am + 32 * (tid >> 6) * (LDA + 1);
    const int t = tid & 63, g = t >> 3, j = 2 * (t & 7);
    product(two, M + 16 * LDA, M + j, 0, 16, g, 8, M + 16 + j);
    __syncthreads();
    product(two, M + 16 * LDA + 16, M + 16 + j, 0, 16, g, 8, M + 16 * LDA + j);
    __syncthreads();
  }
  const std::integral_constant<int, 4> four;
  {  // X = A21 T11 -> the unused upper-right block; a warp takes eight columns, T11 is zero above its diagonal
    const int j = 8 * warp + 2 * (lane & 3);
    product(four, Am + 32 * LDA, Am + j, 8 * warp, 32, lane >> 2, 8, Am + 32 + j);
  }
  __syncthreads();
  {  // T21 = T22 X -> over A21 (nothing reads A21 any more); a warp takes eight rows
    const int j = 2 * (lane & 15);
    product(four, Am + 32 * LDA + 32, Am + 32 + j, 0, 8 * warp + 8, 8 * warp + (lane >> 4), 2, Am + 32 * LDA + j);
  }
  __syncthreads();
}
// This thread's units of the bf16 operand images of T and T diag(beta) (the upper triangle reads as zero).
__device__ __forceinline__ void load_inverse_images(const float* Am, const float* bet, uint4 (&timg)[4], uint4 (&tbimg)[4]) {
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int u = threadIdx.x + 128 * m, i = urow8(u), c8 = ucol8(u);
    const float4 a0 = *reinterpret_cast<const float4*>(Am + i * LDA + 8 * c8);
    const float4 a1 = *reinterpret_cast<const float4*>(Am + i * LDA + 8 * c8 + 4);
    float e[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, eb[8];
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      const int mm = 8 * c8 + y;
      e[y] = (mm <= i) ? e[y] : 0.f;
      eb[y] = e[y] * bet[mm];
    }
    timg[m] = make_uint4(tc::pack_bf16(e[0], e[1]), tc::pack_bf16(e[2], e[3]), tc::pack_bf16(e[4], e[5]), tc::pack_bf16(e[6], e[7]));
    tbimg[m] = make_uint4(tc::pack_bf16(eb[0], eb[1]), tc::pack_bf16(eb[2], eb[3]), tc::pack_bf16(eb[4], eb[5]), tc::pack_bf16(eb[6], eb[7]));
  }
}
}  // namespace tcg
using namespace tcg;

// State passes on mma.sync (gdn_chain.cu).  chain_columns: columns of the state per CTA, 0 where the tcgen05 passes are the better
// ones; whole: the images of the state are wanted at their full width (saving forward, backward).  Then the passes, nv columns per
// CTA; maps.k, maps.q as the other kernels use them.
int chain_columns(const TcP& p, bool whole);
mxb_status chain_fwd(const TcP& p, const RowMaps& maps, int nv, cudaStream_t st);
mxb_status chain_bwd(const TcP& p, const RowMaps& maps, int nv, cudaStream_t st);

}  // namespace mxb
