// Gated delta rule, chunked WY/UT form, forward and backward - full-fp32
// CUDA-core path.  Serves fp32 I/O (parity to 1e-4 cannot be met through
// bf16/tf32 tensor-core operands) and any shape the tensor-core path does not
// cover (ragged Dk/Dv, chunk != 64).  Math follows the reference's
// gated_delta_scan_chunked (gpu/ir.cpp:2352-2550):
//
//   gam = cumsum_C(log max(gate,1e-30));  E(x) = exp(clamp(x,-80,0))
//   A   = -(k beta . k^T) * E(gam_i-gam_j) * [i>j];   T = (I-A)^-1
//   u   = T (v beta);  w = T (k beta E(gam));  P = (q k^T) * E(gam_i-gam_j) * [i>=j]
//   per chunk:  v_new = u - w S;  o = (q E(gam)) S + P v_new
//               S <- S E(gam_last) + (k E(gam_last-gam))^T v_new
//
// The backward is hand-derived (the reference differentiates the forward with
// MLX autograd; only the solve has a VJP, tril(T^T dT T^T,-1),
// gpu/gated_delta_cuda_primitive.cpp:104-132, which appears below as dA).
//
// Kernels:
//   gdn_prep_kernel        one CTA per (chunk, b*H+h): gam, T, w, u, P -> workspace
//   gdn_state_fwd_kernel   one CTA per (slab of 4, 8 or 16 columns of Dv, b*H+h), sequential over
//                          chunks: v_new, out, state (columns of Dv are independent)
//   gdn_state_bwd_kernel   same mapping, reverse over chunks: dv_new, dS
//   gdn_chunk_bwd_kernel   one CTA per chunk: dq, dk, dv, dbeta, dgate
//   gdn_recurrent_fwd_kernel  token-by-token recurrence (chunk <= 1,
//                          gated_delta_scan_naive, gpu/ir.cpp:2314-2350)
//
// All products are register-tiled over shared-memory tiles of 64 rows (a chunk, zero-padded) and issue packed
// two-wide FMAs: a chain of fp32 sums either way, with half the issue slots, which the shared-memory loads need.
#include <cuda.h>

#include <cstring>
#include <initializer_list>
#include <type_traits>

#include "common.cuh"
#include "packed.cuh"
#include "tcgen05.cuh"

namespace mxb {

// [B,T,H,D] float32 -> tensor map with boxes of 32 columns x 64 rows, 128-byte swizzle; false if it cannot be made.
bool make_tma_map_f32(CUtensorMap* m, const void* base, int B, int T, int H, int D);

struct GdnP {
  int B, T, H, K, V, C, n, gate_is_log, save;
  int tma;         // the state passes fetch their tiles with the copy engine (float32, Dk % 4 == 0, chunks of 64)
  int vtma;        // the same for v (Dv % 4 == 0)
  int vecK, vecV;  // rows of Dk / Dv elements can be read and written four elements at a time
  const void *q, *k, *v;
  const float *beta, *gate, *h0;
  void* out;
  float* hT;
  const void* dO;
  const float* dhT_in;
  void *dq, *dk, *dv;
  float *dbeta, *dgate, *dh0;
  // workspace, all fp32, indexed by ci = (b*H+h)*n + chunk
  int* status;  // 256-byte header: 5 when a bounded wait gave up
  float *gam;   // [C]
  float *Tm;    // [C,C]  (written when the forward saves for the backward)
  float *w;     // [C,K]
  float *u;     // [C,V]
  float *P;     // [C,C]
  float *hs;    // [V,K]  state at chunk start, transposed
  float *vn;    // [C,V]
  float *dhs;   // [V,K]  dS at chunk end, transposed
  float *dvn;   // [C,V]
  float *e;     // [C,V]  T^T dv_new
  float *z;     // [C,K]  T^T dw
};

__device__ __forceinline__ float log_gate(float g, int gate_is_log) {
  return gate_is_log ? fmaxf(g, kLogGateFloor) : logf(fmaxf(g, kGateFloor));
}

// ---------------------------------------------------------- tiles and products
namespace simt {
constexpr int R = 64;    // tile rows: a chunk, zero-padded
constexpr int LD = 68;   // pitch of [64][64] matrices: rows 16 bytes apart modulo 128, so that eight rows read at the
                         // same column fall into different banks
constexpr int KB = 32;   // contraction elements staged per step
constexpr int LB = KB + 4;

__device__ __forceinline__ ulonglong2 lds2x2(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// Four consecutive elements col .. col+3 of a row of n (zeros past the end).
template <typename IO>
__device__ __forceinline__ float4 ld4(const IO* row, int col, int n, bool vec);
template <>
__device__ __forceinline__ float4 ld4<float>(const float* row, int col, int n, bool vec) {
  if (col >= n) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec) return *reinterpret_cast<const float4*>(row + col);
  return make_float4(row[col], col + 1 < n ? row[col + 1] : 0.f, col + 2 < n ? row[col + 2] : 0.f, col + 3 < n ? row[col + 3] : 0.f);
}
template <>
__device__ __forceinline__ float4 ld4<__nv_bfloat16>(const __nv_bfloat16* row, int col, int n, bool vec) {
  if (col >= n) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec) {
    const uint2 w = *reinterpret_cast<const uint2*>(row + col);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
  return make_float4(to_f32(row[col]), col + 1 < n ? to_f32(row[col + 1]) : 0.f, col + 2 < n ? to_f32(row[col + 2]) : 0.f,
                     col + 3 < n ? to_f32(row[col + 3]) : 0.f);
}
template <typename IO>
__device__ __forceinline__ void st4(IO* row, int col, int n, bool vec, float4 x) {
  if (col >= n) return;
  if (vec) {
    if constexpr (sizeof(IO) == 4) {
      *reinterpret_cast<float4*>(row + col) = x;
    } else {
      __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
      *reinterpret_cast<uint2*>(row + col) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    }
    return;
  }
  row[col] = from_f32<IO>(x.x);
  if (col + 1 < n) row[col + 1] = from_f32<IO>(x.y);
  if (col + 2 < n) row[col + 2] = from_f32<IO>(x.z);
  if (col + 3 < n) row[col + 3] = from_f32<IO>(x.w);
}
__device__ __forceinline__ float4 scale4(float4 x, float s) { return make_float4(x.x * s, x.y * s, x.z * s, x.w * s); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}

// acc[r][c] += sum_k A[ty + 16 r][k] B[tx + 16 c][k]: both operands contiguous along the contraction, the two halves
// of an accumulator take its even and odd elements.
__device__ __forceinline__ void tile_nt(f2 (&acc)[4][4], const float* A, int lda, const float* B, int ldb, int kd) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
  for (int k = 0; k < kd; k += 4) {
    ulonglong2 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = lds2x2(A + (ty + 16 * r) * lda + k);
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = lds2x2(B + (tx + 16 * c) * ldb + k);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        fma2(acc[r][c], a[r].x, b[c].x);
        fma2(acc[r][c], a[r].y, b[c].y);
      }
  }
}
// acc[r][2 g + s] += sum_k A[4 ty + r][k] B[k][64 g + 4 tx + 2 s, +1].  AT: A is stored transposed, [k][i].
template <int NG, bool AT>
__device__ __forceinline__ void tile_nn(f2 (&acc)[4][2 * NG], const float* A, int lda, const float* B, int ldb, int kd) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 2
  for (int k = 0; k < kd; k += 4) {
    float a[4][4];  // [row][k]
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 t = AT ? *reinterpret_cast<const float4*>(A + (k + r) * lda + 4 * ty)
                          : *reinterpret_cast<const float4*>(A + (4 * ty + r) * lda + k);
      if (AT) { a[0][r] = t.x; a[1][r] = t.y; a[2][r] = t.z; a[3][r] = t.w; }
      else { a[r][0] = t.x; a[r][1] = t.y; a[r][2] = t.z; a[r][3] = t.w; }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      ulonglong2 b[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) b[g] = lds2x2(B + (k + kk) * ldb + 64 * g + 4 * tx);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const f2 aa = pack2(a[r][kk], a[r][kk]);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          fma2(acc[r][2 * g], aa, b[g].x);
          fma2(acc[r][2 * g + 1], aa, b[g].y);
        }
      }
    }
  }
}
template <int N>
__device__ __forceinline__ void clear(f2 (&acc)[4][N]) {
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) acc[r][c] = 0ull;
}
template <int NG>
__device__ __forceinline__ float4 acc4(const f2 (&acc)[4][2 * NG], int r, int g) {
  const float2 a = unpack2(acc[r][2 * g]), b = unpack2(acc[r][2 * g + 1]);
  return make_float4(a.x, a.y, b.x, b.y);
}
// Sum over the 16 threads that share the rows of a tile.
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Streaming buffers of the products whose operands come from global memory: two stages of KB contraction elements,
// the next stage's elements in registers while the current one is multiplied.
constexpr int kStageA = R * LB;      // [64][LB]
constexpr int kStageB = KB * 128;    // [KB][128], or [64][LB] for the products along rows
constexpr int kStageFloats = 2 * (kStageA + kStageB);
static_assert(kStageB >= R * LB, "row blocks fit the stage of the wide operand");

// acc += A B^T over kd elements; la(i, k), lb(j, k) give elements k .. k+3 of row i of A, row j of B.
template <typename FA, typename FB>
__device__ __forceinline__ void stream_nt(f2 (&acc)[4][4], float* stage, int kd, FA la, FB lb) {
  float4 ra[2], rb[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int u = threadIdx.x + 256 * m, i = u >> 3, c = 4 * (u & 7);
      ra[m] = la(i, k0 + c);
      rb[m] = lb(i, k0 + c);
    }
  };
  auto put = [&](int buf) {
    float* sA = stage + buf * kStageA;
    float* sB = stage + 2 * kStageA + buf * kStageB;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int u = threadIdx.x + 256 * m, i = u >> 3, c = 4 * (u & 7);
      *reinterpret_cast<float4*>(sA + i * LB + c) = ra[m];
      *reinterpret_cast<float4*>(sB + i * LB + c) = rb[m];
    }
  };
  fetch(0);
  __syncthreads();  // whoever used the stages before is done
  put(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < kd; k0 += KB, buf ^= 1) {
    const bool more = k0 + KB < kd;
    if (more) fetch(k0 + KB);
    tile_nt(acc, stage + buf * kStageA, LB, stage + 2 * kStageA + buf * kStageB, LB, KB);
    if (more) put(buf ^ 1);
    __syncthreads();
  }
}
// acc += A B over kd elements, B streamed: lb(k, j) gives elements j .. j+3 of row k.  A streamed (AM = 0, la(i, k)),
// or a [64][64] matrix in shared memory as it is (AM = 1) or transposed (AM = 2), pitch LD.
template <int NG, int AM, typename FA, typename FB>
__device__ __forceinline__ void stream_nn(f2 (&acc)[4][2 * NG], float* stage, int kd, const float* As, FA la, FB lb) {
  constexpr int NB = 2 * NG;  // units of four per thread in a KB x 64 NG block
  float4 ra[2], rb[NB];
  auto fetch = [&](int k0) {
    if (AM == 0) {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int u = threadIdx.x + 256 * m;
        ra[m] = la(u >> 3, k0 + 4 * (u & 7));
      }
    }
#pragma unroll
    for (int m = 0; m < NB; ++m) {
      const int u = threadIdx.x + 256 * m;
      rb[m] = lb(k0 + u / (16 * NG), 4 * (u % (16 * NG)));
    }
  };
  auto put = [&](int buf) {
    if (AM == 0) {
      float* sA = stage + buf * kStageA;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int u = threadIdx.x + 256 * m;
        *reinterpret_cast<float4*>(sA + (u >> 3) * LB + 4 * (u & 7)) = ra[m];
      }
    }
    float* sB = stage + 2 * kStageA + buf * kStageB;
#pragma unroll
    for (int m = 0; m < NB; ++m) *reinterpret_cast<float4*>(sB + 4 * (threadIdx.x + 256 * m)) = rb[m];
  };
  fetch(0);
  __syncthreads();
  put(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < kd; k0 += KB, buf ^= 1) {
    const bool more = k0 + KB < kd;
    if (more) fetch(k0 + KB);
    const float* sB = stage + 2 * kStageA + buf * kStageB;
    if (AM == 0) tile_nn<NG, false>(acc, stage + buf * kStageA, LB, sB, 64 * NG, KB);
    else if (AM == 1) tile_nn<NG, false>(acc, As + k0, LD, sB, 64 * NG, KB);
    else tile_nn<NG, true>(acc, As + k0 * LD, LD, sB, 64 * NG, KB);
    if (more) put(buf ^ 1);
    __syncthreads();
  }
}
struct NoA { __device__ float4 operator()(int, int) const { return make_float4(0.f, 0.f, 0.f, 0.f); } };
}  // namespace simt

// ------------------------------------------------------------ state passes
// The sequential passes: one chunk after the other, so the time of a chunk is what counts.  A CTA owns W columns of
// the state (columns are independent), W as small as still fits the CTAs on the SMs at once.  What bounds a chunk are
// the shared-memory reads of the products and the eight warps an SM that hide them (40 to 43 % of that pipe, 28 to 31 %
// of the issue slots), so every thread computes 4 x 4 outputs (eight loaded values per sixteen multiply-adds) over a part
// of the contraction, and the parts (32 / W of them for 128 rows) are added through shared memory in a fixed order.  One
// output per thread and 16-column slabs, operands by one cp.async per 16 bytes:
// 8.2 us a chunk at Dk = 64 (6.6 k of 16.4 k cycles went into issuing the copies; one bulk copy per row still took
// its warp 2.2 k); now a tile is two or four tensor copies issued by one thread as soon as the tile it replaces has
// been read.
//
// A thread's 4 x 4 outputs of a product along rows: rows ty + NR r, columns tx + NCG c.
template <int W, int NR>
struct SlabMap {
  static constexpr int NCG = W / 4;             // column groups
  static constexpr int PER = NR * NCG;          // threads that share a part of the contraction
  static constexpr int PITCH = W == 16 ? 20 : W + 1;  // of a row of partial sums (few bank conflicts both ways)
};
// The operand tiles that travel (w, q, k, P) lie as the copy engine writes boxes of 32 floats with 128-byte swizzle:
// slabs of 32 columns, the 16-byte unit within a row XORed with the row's position in its group of eight, so that
// eight rows read at the same column, or eight units of one row, come from different banks.  Unit u of row i:
template <int ROWS>
__device__ __forceinline__ int slab_unit(int i, int u) { return (u >> 3) * (ROWS * 32) + i * 32 + (((u & 7) ^ (i & 7)) << 2); }

// part[s][ty + NR r][tx + NCG c] = sum over the s-th part of the contraction of A[row][k] B[col][k]; `t` < SP * PER
template <int W, int NR, int SP, int ROWS, int KD>
__device__ __forceinline__ void slab_nt(float* part, const float* A, const float* B, int ldb, int t) {
  using namespace simt;
  using M = SlabMap<W, NR>;
  const int tx = t % M::NCG, ty = (t / M::NCG) % NR, s = t / M::PER;
  constexpr int LEN = KD / SP / 4;  // units of four per part
  f2 acc[4][4];
  clear(acc);
  const float* b0 = B + tx * ldb;
#pragma unroll 2
  for (int x = 0; x < LEN; ++x) {
    const int u = s * LEN + x;
    const float* a0 = A + slab_unit<ROWS>(ty, u);  // (the rows of a thread are a multiple of eight apart)
    ulonglong2 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = lds2x2(a0 + NR * 32 * r);
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] = lds2x2(b0 + M::NCG * c * ldb + 4 * u);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        fma2(acc[r][c], a[r].x, b[c].x);
        fma2(acc[r][c], a[r].y, b[c].y);
      }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      part[s * 4 * NR * M::PITCH + (ty + NR * r) * M::PITCH + tx + M::NCG * c] = sum2(acc[r][c]);
}
// part[s][4 tx + c][kk] = sum over the s-th part of the 64 rows i of A[i][kk] B[i][4 tx + c]; t < 128
template <int W, int KP, int ROWS>
__device__ __forceinline__ void slab_tn(float* part, const float* A, const float* B, int t) {
  using namespace simt;
  constexpr int LK = KP + 4, NCG = W / 4, PER = NCG * (KP / 4), SP = 128 / PER, LEN = R / SP;
  const int tx = t % NCG, kg = (t / NCG) % (KP / 4), s = t / PER;
  f2 acc[4][2];  // [column][pair of state rows]
  clear(acc);
  const float* b0 = B + s * LEN * W + 4 * tx;
#pragma unroll 4
  for (int i = 0; i < LEN; ++i) {
    const ulonglong2 a = lds2x2(A + slab_unit<ROWS>(s * LEN + i, kg));
    const float4 b = *reinterpret_cast<const float4*>(b0 + i * W);
    const f2 bb[4] = {pack2(b.x, b.x), pack2(b.y, b.y), pack2(b.z, b.z), pack2(b.w, b.w)};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      fma2(acc[c][0], a.x, bb[c]);
      fma2(acc[c][1], a.y, bb[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<ulonglong2*>(part + (s * W + 4 * tx + c) * LK + 4 * kg) = make_ulonglong2(acc[c][0], acc[c][1]);
}
constexpr int kSlabScalars = 2 * simt::R + 4;  // E(gam), E(gam_last - gam), E(gam_last)

// Tensor maps of the tiles: boxes of 32 columns x 64 rows; rows past the end of a sequence and columns past Dk arrive as
// zeros.
struct alignas(64) SlabMaps {
  CUtensorMap w, q, k, P;  // P: v in the prep kernel
};
// Rows 0 .. 63 of a tile of KP columns by the threads themselves (bf16 rows are widened), zeros past `rows` and n.
template <typename IO, int KP, int ROWS, typename F>
__device__ __forceinline__ void slab_copy(float* dst, int rows, int n, int vec, F rowptr) {
  for (int u = threadIdx.x; u < simt::R * (KP / 4); u += 256) {
    const int i = u / (KP / 4), c4 = u % (KP / 4);
    *reinterpret_cast<float4*>(dst + slab_unit<ROWS>(i, c4)) =
        i < rows ? simt::ld4(rowptr(i), 4 * c4, n, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
// A [C][C] matrix of the workspace (what lies outside stays zero from the start).
__device__ __forceinline__ void slab_square(float* dst, const float* src, int C) {
  for (int u = threadIdx.x; u < C * C; u += 256) {
    const int i = u / C, j = u % C;
    dst[slab_unit<simt::R>(i, j >> 2) + (j & 3)] = src[u];
  }
}

// ------------------------------------------------------------------ prep
// One chunk, a chain of dependent steps: copies -> [k;q] k^T -> triangular inverse -> (T beta) v, (T beta)(E(gam) k).
// k, q and v are requested at once and stay in shared memory in the swizzled layout of their copies, k is scaled in
// place beside the inverse; 82 KB, two CTAs per SM.  (Streaming every product's operands in steps of 32 exposed the
// latency of global memory a dozen times: 18.8 us for 32 chunks of 64 / 64 columns on an empty GPU.)
template <int KP>
struct PrepF32 {
  static constexpr int VC = 128;                         // columns of v at a time
  static constexpr int kv = KP == 64 ? simt::R * VC : 0; // floats of v's own tile; 128 columns of v go over q
  static constexpr int smem = 4 * (2 * simt::R * KP + kv + simt::R * simt::LD + 4 * simt::R) + 64 + 1024;
};

// acc[r][2 g + s] += sum_{m < 4 ty + 4} A[4 ty + r][m] B[m][64 g + 4 tx + 2 s, +1], A lower triangular, B swizzled
template <int NG>
__device__ __forceinline__ void prep_product(f2 (&acc)[4][2 * NG], const float* A, const float* B) {
  using namespace simt;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 2
  for (int m = 0; m < 4 * ty + 4; m += 4) {
    float a[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 t = *reinterpret_cast<const float4*>(A + (4 * ty + r) * LD + m);
      a[r][0] = t.x; a[r][1] = t.y; a[r][2] = t.z; a[r][3] = t.w;
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      ulonglong2 b[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) b[g] = lds2x2(B + slab_unit<R>(m + y, 16 * g + tx));
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const f2 aa = pack2(a[r][y], a[r][y]);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          fma2(acc[r][2 * g], aa, b[g].x);
          fma2(acc[r][2 * g + 1], aa, b[g].y);
        }
      }
    }
  }
}

template <typename IO, int KP>
__global__ void __launch_bounds__(256, 2) gdn_prep_kernel(GdnP p, const __grid_constant__ SlabMaps maps) {
  begin_dependent();
  using namespace simt;
  extern __shared__ float smem_raw[];
  float* Ks = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(smem_raw) + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u));
  float* Qs = Ks + R * KP;
  float* Vs = KP == 64 ? Qs + R * KP : Qs;  // 128 columns of v
  float* Am = Qs + R * KP + PrepF32<KP>::kv;  // [64][LD]  A, then T, then T diag(beta)
  float* gam = Am + R * LD;
  float* bet = gam + R;
  float* dd = bet + R;  // E(gam)
  uint64_t* bar = reinterpret_cast<uint64_t*>(dd + 2 * R);  // [0] k, q; [1] v
  const int C = p.C, K = p.K, V = p.V;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31;
  const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H, t0 = c * C;
  const int imax = min(C, p.T - t0);
  const size_t ci = (size_t)bh * p.n + c;
  const IO* q = static_cast<const IO*>(p.q);
  const IO* k = static_cast<const IO*>(p.k);
  const IO* v = static_cast<const IO*>(p.v);
  auto row = [&](int i) { return ((size_t)(b * p.T + t0 + i) * p.H + h); };
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool tma = p.tma, vtma = p.vtma;
  auto load_v = [&](int j0) {  // columns j0 .. of v; columns past Dv are not read by anyone
    if (vtma) {
      if (tid == 0) {
        const int nx = min(4, (V - j0 + 31) / 32);
        tc::mbar_expect_tx(bar + 1, nx * R * 32 * 4);
        for (int x = 0; x < nx; ++x) tc::tma_load_4d(tc::smem_u32(Vs + x * 2048), &maps.P, j0 + 32 * x, h, t0, b, bar + 1);
      }
    } else {
      for (int u = tid; u < R * 32; u += 256) {
        const int i = u >> 5, c4 = u & 31;
        *reinterpret_cast<float4*>(Vs + slab_unit<R>(i, c4)) = i < imax ? ld4(v + row(i) * V, j0 + 4 * c4, V, p.vecV) : zero;
      }
    }
  };
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(bar + 1, 1);
    tc::mbar_fence_init();
    if (tma) {
      tc::mbar_expect_tx(bar, 2 * R * KP * 4);
      for (int x = 0; x < KP / 32; ++x) {
        tc::tma_load_4d(tc::smem_u32(Ks + x * 2048), &maps.k, 32 * x, h, t0, b, bar);
        tc::tma_load_4d(tc::smem_u32(Qs + x * 2048), &maps.q, 32 * x, h, t0, b, bar);
      }
    }
  }
  if (!tma) {
    slab_copy<IO, KP, R>(Ks, imax, K, p.vecK, [&](int i) { return k + row(i) * K; });
    slab_copy<IO, KP, R>(Qs, imax, K, p.vecK, [&](int i) { return q + row(i) * K; });
  }
  if (KP == 64) load_v(0);
  if (c == 0 && bh == 0 && tid >= 64 && tid < 128) p.status[tid - 64] = 0;
  if (tid >= 32 && tid < 64) {
    // Inclusive cumulative sum of the log gate, one step after the other: neighbouring sums then differ by a gate and ONE
    // rounding, and it is differences of near sums that E(gam_i - gam_j) is large for.  (The rounding of these sums is the
    // error of the whole scan.  Summed by a tree across the lanes it was 1.7 times as large; the chain of 64 additions runs
    // beside the copies of k and q.)
    const int i0 = 2 * lane, i1 = i0 + 1;
    const float b0 = i0 < imax ? p.beta[row(i0)] : 0.f, b1 = i1 < imax ? p.beta[row(i1)] : 0.f;
    gam[i0] = i0 < imax ? log_gate(p.gate[row(i0)], p.gate_is_log) : 0.f;
    gam[i1] = i1 < imax ? log_gate(p.gate[row(i1)], p.gate_is_log) : 0.f;
    __syncwarp();
    if (lane == 0) {
      float4 g[R / 4];
#pragma unroll
      for (int x = 0; x < R / 4; ++x) g[x] = *reinterpret_cast<const float4*>(gam + 4 * x);
      float s = 0.f;
#pragma unroll
      for (int x = 0; x < R / 4; ++x) {
        g[x].x = s += g[x].x;
        g[x].y = s += g[x].y;
        g[x].z = s += g[x].z;
        g[x].w = s += g[x].w;
        *reinterpret_cast<float4*>(gam + 4 * x) = g[x];
      }
    }
    __syncwarp();
    const float c0 = gam[i0], c1 = gam[i1];
    bet[i0] = b0; bet[i1] = b1;
    dd[i0] = exp_nonpos_precise(c0); dd[i1] = exp_nonpos_precise(c1);
    if (i0 < C) p.gam[ci * C + i0] = c0;
    if (i1 < C) p.gam[ci * C + i1] = c1;
  }
  __syncthreads();
  bool ok = !tma || tc::mbar_wait(bar, 0);
  {  // k k^T and q k^T: rows ty + 16 r of both, columns tx + 16 x, lower 16 x 16 blocks only
    f2 acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[r][x] = 0ull;
#pragma unroll 2
    for (int u = 0; u < KP / 4; ++u) {
      const float* a0 = Ks + slab_unit<R>(ty, u);
      const float* b0 = Ks + slab_unit<R>(tx, u);
      ulonglong2 bb[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) bb[x] = lds2x2(b0 + 16 * 32 * x);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const ulonglong2 a = lds2x2(a0 + (r >> 2) * R * KP + 16 * 32 * (r & 3));
#pragma unroll
        for (int x = 0; x <= (r & 3); ++x) {
          fma2(acc[r][x], a.x, bb[x].x);
          fma2(acc[r][x], a.y, bb[x].y);
        }
      }
    }
    float* P = p.P + ci * C * C;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int i = ty + 16 * r, j = tx + 16 * x;
        const float e = x <= r ? exp_nonpos_precise(gam[i] - gam[j]) : 0.f;
        Am[i * LD + j] = (i > j) ? -bet[i] * sum2(acc[r][x]) * e : 0.f;
        if (i < C && j < C) P[i * C + j] = (i >= j) ? sum2(acc[4 + r][x]) * e : 0.f;
      }
  }
  tc::fence_async_smem();
  __syncthreads();  // A is in place, q has been read
  if (KP != 64) load_v(0);
  // T = (I - A)^-1 in place: the two 32 x 32 diagonal blocks by forward substitution (thread = block and column, the
  // column in registers) while the other threads scale k to E(gam) k, then the off-diagonal block T21 = T22 (A21 T11)
  // as two 32^3 products over all threads.
  {
    float Tc[32];
    const int cc = tid & 31, r0 = 32 * ((tid >> 5) & 1);
    if (tid < R) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float* arow = Am + (r0 + i) * LD + r0;
        float s0 = (i == cc) ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
        for (int j = 0; j + 1 < i; j += 2) {
          s0 = fmaf(arow[j], Tc[j], s0);
          s1 = fmaf(arow[j + 1], Tc[j + 1], s1);
        }
        if (i & 1) s0 = fmaf(arow[i - 1], Tc[i - 1], s0);
        Tc[i] = (i < cc) ? 0.f : s0 + s1;
      }
    } else {
      for (int u = tid - R; u < R * (KP / 4); u += 192) {
        const int i = u / (KP / 4);
        float4* x = reinterpret_cast<float4*>(Ks + slab_unit<R>(i, u % (KP / 4)));
        *x = scale4(*x, dd[i]);
      }
    }
    __syncthreads();
    if (tid < R) {
#pragma unroll
      for (int i = 0; i < 32; ++i) Am[(r0 + i) * LD + r0 + cc] = Tc[i];
    }
    __syncthreads();
    const int i2 = tid >> 3, jb = (tid & 7) * 4;
    float4 x = zero;
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {  // X = A21 T11 -> the unused upper-right block
      const float a = Am[(32 + i2) * LD + m];
      const float4 t = *reinterpret_cast<const float4*>(Am + m * LD + jb);
      x = make_float4(fmaf(a, t.x, x.x), fmaf(a, t.y, x.y), fmaf(a, t.z, x.z), fmaf(a, t.w, x.w));
    }
    *reinterpret_cast<float4*>(Am + i2 * LD + 32 + jb) = x;
    __syncthreads();
    float4 y = zero;
#pragma unroll 8
    for (int m = 0; m < 32; ++m) {  // T21 = T22 X -> over A21
      const float a = Am[(32 + i2) * LD + 32 + m];
      const float4 t = *reinterpret_cast<const float4*>(Am + m * LD + 32 + jb);
      y = make_float4(fmaf(a, t.x, y.x), fmaf(a, t.y, y.y), fmaf(a, t.z, y.z), fmaf(a, t.w, y.w));
    }
    __syncthreads();
    *reinterpret_cast<float4*>(Am + (32 + i2) * LD + jb) = y;
    *reinterpret_cast<float4*>(Am + i2 * LD + 32 + jb) = zero;  // the upper-right block of T
    __syncthreads();
  }
  for (int u = tid; u < R * R; u += 256) {  // T leaves for the backward; its columns are scaled by beta
    const int i = u >> 6, j = u & 63;
    const float t = Am[i * LD + j];
    if (p.save && i < C && j < C) p.Tm[ci * C * C + i * C + j] = t;
    Am[i * LD + j] = t * bet[j];
  }
  __syncthreads();
  {  // w
    constexpr int NG = KP / 64;
    f2 acc[4][2 * NG];
    clear(acc);
    prep_product<NG>(acc, Am, Ks);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int g = 0; g < NG; ++g)
        if (4 * ty + r < C) st4(p.w + (ci * C + 4 * ty + r) * K, 64 * g + 4 * tx, K, p.vecK, acc4<NG>(acc, r, g));
  }
  for (int j0 = 0, it = 0; j0 < V; j0 += 128, ++it) {  // u
    if (it > 0) {
      tc::fence_async_smem();
      __syncthreads();
      load_v(j0);
    }
    if (vtma) ok = tc::mbar_wait(bar + 1, it & 1) && ok;
    else __syncthreads();
    auto product = [&](auto ng) {
      constexpr int NG = decltype(ng)::value;
      f2 acc[4][2 * NG];
      clear(acc);
      prep_product<NG>(acc, Am, Vs);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int g = 0; g < NG; ++g)
          if (4 * ty + r < C) st4(p.u + (ci * C + 4 * ty + r) * V, j0 + 64 * g + 4 * tx, V, p.vecV, acc4<NG>(acc, r, g));
    };
    if (V - j0 <= 64) product(std::integral_constant<int, 1>{});
    else product(std::integral_constant<int, 2>{});
  }
  if (!ok && tid == 0) atomicExch(p.status, 5);
}

// ----------------------------------------------------------- state passes: slabs
// Floats of the partial sums: 128 rows of W columns in 32 / W parts (the products of the second step need less).
template <int W>
constexpr int kSlabPart = 32 / W * 128 * SlabMap<W, 16>::PITCH;
template <int W, int KP>
constexpr int state_fwd_smem() {
  return 4 * (192 * KP + simt::R * simt::R + W * (KP + 4) + W * simt::LD + simt::R * W + 2 * kSlabScalars + kSlabPart<W>) + 64 + 1024;
}
template <int W, int KP>
constexpr int state_bwd_smem() {
  return 4 * (192 * KP + simt::R * simt::R + W * (KP + 4) + 3 * simt::R * W + 2 * kSlabScalars + kSlabPart<W>) + 64 + 1024;
}
// Decay factors of one chunk from its in-chunk cumulative log decay g (lane's own) and gl (the last).
__device__ __forceinline__ void slab_scalars(float* s, float g, float gl) {
  const int tid = threadIdx.x;
  if (tid < simt::R) {
    s[tid] = exp_nonpos_precise(g);
    s[simt::R + tid] = exp_nonpos_precise(gl - g);
    if (tid == 0) s[2 * simt::R] = exp_nonpos_precise(gl);
  }
}
// State slab (transposed, pitch LK) <-> [K][V] tensor columns j0 .. j0+W-1.
template <int W, int KP>
__device__ __forceinline__ void slab_state_in(float* St, const float* src, int K, int V, int j0) {
  for (int u = threadIdx.x; u < W * KP; u += 256) {
    const int j = u % W, kk = u / W;
    St[j * (KP + 4) + kk] = (src && kk < K && j0 + j < V) ? src[(size_t)kk * V + j0 + j] : 0.f;
  }
}
template <int W, int KP>
__device__ __forceinline__ void slab_state_out(const float* St, float* dst, int K, int V, int j0) {
  for (int u = threadIdx.x; u < W * KP; u += 256) {
    const int j = u % W, kk = u / W;
    if (kk < K && j0 + j < V) dst[(size_t)kk * V + j0 + j] = St[j * (KP + 4) + kk];
  }
}
// The same slab as rows of the transposed states [V][K] kept per chunk.
template <int W, int KP>
__device__ __forceinline__ void slab_state_keep(const float* St, float* dst, int K, int V, int vec, int j0) {
  for (int u = threadIdx.x; u < W * KP / 4; u += 256) {
    const int j = u / (KP / 4), kk = 4 * (u % (KP / 4));
    if (j0 + j < V) simt::st4(dst + (size_t)(j0 + j) * K, kk, K, vec, *reinterpret_cast<const float4*>(St + j * (KP + 4) + kk));
  }
}
// State <- L state + partial sums (NP of them), and the copy kept for chunk kernels where `keep` is not null.
template <int W, int KP, int NP>
__device__ __forceinline__ void slab_state_step(float* St, const float* part, float L, float* keep, int K, int V, int vec, int j0) {
  constexpr int LK = KP + 4;
  for (int u = threadIdx.x; u < W * KP / 4; u += 256) {
    const int j = u / (KP / 4), kk = 4 * (u % (KP / 4));
    float4* own = reinterpret_cast<float4*>(St + j * LK + kk);
    float4 x = simt::scale4(*own, L);
#pragma unroll
    for (int s = 0; s < NP; ++s) {
      const float4 t = *reinterpret_cast<const float4*>(part + (s * W + j) * LK + kk);
      x = make_float4(x.x + t.x, x.y + t.y, x.z + t.z, x.w + t.w);
    }
    *own = x;
    if (keep && j0 + j < V) simt::st4(keep + (size_t)(j0 + j) * K, kk, K, vec, x);
  }
}
template <int W>
__device__ __forceinline__ float slab_sum(const float* part, int rows, int row, int col) {
  float v = 0.f;
#pragma unroll
  for (int s = 0; s < 32 / W; ++s) v += part[(s * rows + row) * SlabMap<W, 16>::PITCH + col];
  return v;
}

// v_new = u - w S;  o = E(gam) (q S) + P v_new;  S <- E(gam_last) S + (k r)^T v_new
template <typename IO, int W, int KP>
__global__ void __launch_bounds__(256, 1) gdn_state_fwd_kernel(GdnP p, const __grid_constant__ SlabMaps maps) {
  begin_dependent();
  using namespace simt;
  constexpr int LK = KP + 4, SP = 32 / W, SPK = 2048 / (W * KP), PITCH = SlabMap<W, 16>::PITCH;
  extern __shared__ float smem_raw[];
  float* Wq = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(smem_raw) + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u));
                                 // slabs of [128 rows][32]: w rows, then q rows
  float* Ks = Wq + 128 * KP;     // slabs of [64][32]
  float* Ps = Ks + R * KP;       // slabs of [64][32]
  float* St = Ps + R * R;        // [W][LK]  S^T
  float* Vt = St + W * LK;       // [W][LD]  v_new^T
  float* Vr = Vt + W * LD;       // [64][W]  r_i v_new
  float* sc = Vr + R * W;        // x2 decay factors of a chunk
  float* part = sc + 2 * kSlabScalars;
  float* partK = part + SP * R * PITCH;  // beside the 64 rows of P v_new
  uint64_t* bar = reinterpret_cast<uint64_t*>(part + kSlabPart<W>);  // [0] w, q; [1] k, P
  const int C = p.C, K = p.K, V = p.V;
  const int tid = threadIdx.x;
  const int bh = blockIdx.y, b = bh / p.H, h = bh % p.H, j0 = blockIdx.x * W;
  const IO* q = static_cast<const IO*>(p.q);
  const IO* k = static_cast<const IO*>(p.k);
  IO* out = static_cast<IO*>(p.out);
  auto row = [&](int c, int i) { return ((size_t)(b * p.T + c * C + i) * p.H + h); };
  const bool tma = p.tma;
  auto load_wq = [&](int c) {
    if (c >= p.n) return;
    if (tma) {  // one thread per tensor issues, in different warps
      if (tid == 0) {
        tc::mbar_expect_tx(bar, 128 * KP * 4);
        for (int x = 0; x < KP / 32; ++x) tc::tma_load_4d(tc::smem_u32(Wq + x * 4096), &maps.w, 32 * x, 0, (bh * p.n + c) * R, 0, bar);
      } else if (tid == 32) {
        for (int x = 0; x < KP / 32; ++x) tc::tma_load_4d(tc::smem_u32(Wq + x * 4096 + 2048), &maps.q, 32 * x, h, c * R, b, bar);
      }
    } else {
      const float* w = p.w + ((size_t)bh * p.n + c) * C * K;
      slab_copy<float, KP, 128>(Wq, C, K, p.vecK, [&](int i) { return w + i * K; });
      slab_copy<IO, KP, 128>(Wq + 2048, min(C, p.T - c * C), K, p.vecK, [&](int i) { return q + row(c, i) * K; });
    }
  };
  auto load_kp = [&](int c) {
    if (c >= p.n) return;
    if (tma) {
      if (tid == 64) {
        tc::mbar_expect_tx(bar + 1, R * (KP + R) * 4);
        for (int x = 0; x < KP / 32; ++x) tc::tma_load_4d(tc::smem_u32(Ks + x * 2048), &maps.k, 32 * x, h, c * R, b, bar + 1);
      } else if (tid == 96) {
        for (int x = 0; x < 2; ++x) tc::tma_load_4d(tc::smem_u32(Ps + x * 2048), &maps.P, 32 * x, 0, (bh * p.n + c) * R, 0, bar + 1);
      }
    } else {
      slab_copy<IO, KP, R>(Ks, min(C, p.T - c * C), K, p.vecK, [&](int i) { return k + row(c, i) * K; });
      slab_square(Ps, p.P + ((size_t)bh * p.n + c) * C * C, C);
    }
  };
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(bar + 1, 1);
    tc::mbar_fence_init();
  }
  if (C < R)
    for (int u = tid; u < R * R; u += 256) Ps[u] = 0.f;
  slab_state_in<W, KP>(St, p.h0 ? p.h0 + (size_t)bh * K * V : nullptr, K, V, j0);
  const float* gam = p.gam + (size_t)bh * p.n * C;
  float gl = gam[C - 1], g = tid < C ? gam[tid] : gl;
  slab_scalars(sc, g, gl);
  tc::fence_async_smem();
  __syncthreads();
  load_wq(0);
  load_kp(0);
  if (p.save) slab_state_keep<W, KP>(St, p.hs + (size_t)bh * p.n * V * K, K, V, p.vecK, j0);

  bool ok = true;
  for (int c = 0; c < p.n; ++c) {
    const size_t ci = (size_t)bh * p.n + c;
    const float* s = sc + (c & 1) * kSlabScalars;
    const int imax = min(C, p.T - c * C);
    float un[W / 4], oq[W / 4];  // this thread's elements of u (fetched ahead of their use) and of E(gam) q S
#pragma unroll
    for (int x = 0; x < W / 4; ++x) {
      const int i = (tid + 256 * x) / W, jv = j0 + (tid + 256 * x) % W;
      un[x] = (i < C && jv < V) ? p.u[(ci * C + i) * V + jv] : 0.f;
    }
    if (c + 1 < p.n) {
      gl = gam[(c + 2) * C - 1];
      g = tid < C ? gam[(c + 1) * C + tid] : gl;
    }
    if (tma) ok = tc::mbar_wait(bar, c & 1);
    ok = __syncthreads_and(ok);  // w, q, the state and the decay factors are in place
    if (!ok) break;
    slab_nt<W, 32, SP, 128, KP>(part, Wq, St, LK, tid);
    tc::fence_async_smem();
    __syncthreads();
    load_wq(c + 1);
#pragma unroll
    for (int x = 0; x < W / 4; ++x) {
      const int i = (tid + 256 * x) / W, j = (tid + 256 * x) % W;
      const float val = un[x] - slab_sum<W>(part, 128, i, j);
      oq[x] = s[i] * slab_sum<W>(part, 128, R + i, j);
      Vt[j * LD + i] = val;
      Vr[i * W + j] = val * s[R + i];
      if (p.save && i < C && j0 + j < V) p.vn[(ci * C + i) * V + j0 + j] = val;
    }
    if (tma) ok = tc::mbar_wait(bar + 1, c & 1);
    ok = __syncthreads_and(ok);  // v_new, k and P are in place
    if (!ok) break;
    if (tid < 128) slab_nt<W, 16, SP, R, R>(part, Ps, Vt, LD, tid);
    else slab_tn<W, KP, R>(partK, Ks, Vr, tid - 128);
    tc::fence_async_smem();
    __syncthreads();
    load_kp(c + 1);
#pragma unroll
    for (int x = 0; x < W / 4; ++x) {
      const int i = (tid + 256 * x) / W, j = (tid + 256 * x) % W;
      if (i < imax && j0 + j < V) out[row(c, i) * V + j0 + j] = from_f32<IO>(oq[x] + slab_sum<W>(part, R, i, j));
    }
    slab_state_step<W, KP, SPK>(St, partK, s[2 * R], p.save && c + 1 < p.n ? p.hs + (ci + 1) * V * K : nullptr, K, V, p.vecK, j0);
    slab_scalars(sc + ((c + 1) & 1) * kSlabScalars, g, gl);
  }
  if (!ok && tid == 0) atomicExch(p.status, 5);
  if (p.hT && ok) {
    __syncthreads();
    slab_state_out<W, KP>(St, p.hT + (size_t)bh * K * V, K, V, j0);
  }
}

// dv_new = P^T dO + r (k dS);  dS <- E(gam_last) dS + (q E(gam))^T dO - w^T dv_new, chunks in reverse.
template <typename IO, int W, int KP>
__global__ void __launch_bounds__(256, 1) gdn_state_bwd_kernel(GdnP p, const __grid_constant__ SlabMaps maps) {
  begin_dependent();
  using namespace simt;
  constexpr int LK = KP + 4, SP = 32 / W, SPK = 2048 / (W * KP), PITCH = SlabMap<W, 16>::PITCH;
  extern __shared__ float smem_raw[];
  float* Ks = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(smem_raw) + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u));
                                 // slabs of [64][32], the four tiles
  float* Qs = Ks + R * KP;
  float* Ws = Qs + R * KP;
  float* Ps = Ws + R * KP;
  float* St = Ps + R * R;        // [W][LK]   dS^T
  float* Os = St + W * LK;       // [64][W]   dO
  float* Od = Os + R * W;        // [64][W]   E(gam_i) dO
  float* Vn = Od + R * W;        // [64][W]   -dv_new
  float* sc = Vn + R * W;        // x2 decay factors of a chunk
  float* part = sc + 2 * kSlabScalars;
  float* partP = part + SP * R * PITCH;        // P^T dO beside k dS
  float* partW = part + SPK * W * LK;          // w^T dv_new beside q^T dO
  uint64_t* bar = reinterpret_cast<uint64_t*>(part + kSlabPart<W>);  // [0] k, P; [1] q, w
  static_assert(2 * SPK * W * LK <= kSlabPart<W> && SP * (R * PITCH + W * LD) <= kSlabPart<W>, "partial sums of both steps");
  const int C = p.C, K = p.K, V = p.V;
  const int tid = threadIdx.x;
  const int bh = blockIdx.y, b = bh / p.H, h = bh % p.H, j0 = blockIdx.x * W;
  const IO* q = static_cast<const IO*>(p.q);
  const IO* k = static_cast<const IO*>(p.k);
  const IO* dO = static_cast<const IO*>(p.dO);
  auto row = [&](int c, int i) { return ((size_t)(b * p.T + c * C + i) * p.H + h); };
  const bool tma = p.tma;
  auto load_kp = [&](int c) {
    if (c < 0) return;
    if (tma) {
      if (tid == 0) {
        tc::mbar_expect_tx(bar, R * (KP + R) * 4);
        for (int x = 0; x < KP / 32; ++x) tc::tma_load_4d(tc::smem_u32(Ks + x * 2048), &maps.k, 32 * x, h, c * R, b, bar);
      } else if (tid == 32) {
        for (int x = 0; x < 2; ++x) tc::tma_load_4d(tc::smem_u32(Ps + x * 2048), &maps.P, 32 * x, 0, (bh * p.n + c) * R, 0, bar);
      }
    } else {
      slab_copy<IO, KP, R>(Ks, min(C, p.T - c * C), K, p.vecK, [&](int i) { return k + row(c, i) * K; });
      slab_square(Ps, p.P + ((size_t)bh * p.n + c) * C * C, C);
    }
  };
  auto load_qw = [&](int c) {
    if (c < 0) return;
    if (tma) {
      if (tid == 64) {
        tc::mbar_expect_tx(bar + 1, 2 * R * KP * 4);
        for (int x = 0; x < KP / 32; ++x) tc::tma_load_4d(tc::smem_u32(Qs + x * 2048), &maps.q, 32 * x, h, c * R, b, bar + 1);
      } else if (tid == 96) {
        for (int x = 0; x < KP / 32; ++x) tc::tma_load_4d(tc::smem_u32(Ws + x * 2048), &maps.w, 32 * x, 0, (bh * p.n + c) * R, 0, bar + 1);
      }
    } else {
      const float* w = p.w + ((size_t)bh * p.n + c) * C * K;
      slab_copy<IO, KP, R>(Qs, min(C, p.T - c * C), K, p.vecK, [&](int i) { return q + row(c, i) * K; });
      slab_copy<float, KP, R>(Ws, C, K, p.vecK, [&](int i) { return w + i * K; });
    }
  };
  const float* gam = p.gam + (size_t)bh * p.n * C;
  // this thread's elements of dO and the log decay of their rows, fetched a chunk ahead
  float o[W / 4], go[W / 4], gl, g;
  auto fetch = [&](int c) {
    const int rows = min(C, p.T - c * C);
    gl = gam[(c + 1) * C - 1];
    g = tid < C ? gam[c * C + tid] : gl;
#pragma unroll
    for (int x = 0; x < W / 4; ++x) {
      const int i = (tid + 256 * x) / W, jv = j0 + (tid + 256 * x) % W;
      o[x] = (i < rows && jv < V) ? to_f32(dO[row(c, i) * V + jv]) : 0.f;
      go[x] = gam[c * C + min(i, C - 1)];
    }
  };
  auto put = [&](int c) {
    slab_scalars(sc + (c & 1) * kSlabScalars, g, gl);
#pragma unroll
    for (int x = 0; x < W / 4; ++x) {
      const int i = (tid + 256 * x) / W, j = (tid + 256 * x) % W;
      Os[i * W + j] = o[x];
      Od[i * W + j] = o[x] * exp_nonpos_precise(go[x]);
    }
  };
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(bar + 1, 1);
    tc::mbar_fence_init();
  }
  if (C < R)
    for (int u = tid; u < R * R; u += 256) Ps[u] = 0.f;
  slab_state_in<W, KP>(St, p.dhT_in ? p.dhT_in + (size_t)bh * K * V : nullptr, K, V, j0);
  fetch(p.n - 1);
  put(p.n - 1);
  tc::fence_async_smem();
  __syncthreads();
  load_kp(p.n - 1);
  load_qw(p.n - 1);
  slab_state_keep<W, KP>(St, p.dhs + ((size_t)bh * p.n + p.n - 1) * V * K, K, V, p.vecK, j0);

  bool ok = true;
  for (int c = p.n - 1; c >= 0; --c) {
    const size_t ci = (size_t)bh * p.n + c;
    const float* s = sc + (c & 1) * kSlabScalars;
    const uint32_t ph = (p.n - 1 - c) & 1;
    if (c > 0) fetch(c - 1);
    if (tma) ok = tc::mbar_wait(bar, ph);
    ok = __syncthreads_and(ok);  // k, P, dO, dS and the decay factors are in place
    if (!ok) break;
    if (tid < 128) slab_nt<W, 16, SP, R, KP>(part, Ks, St, LK, tid);
    else slab_tn<W, R, R>(partP, Ps, Os, tid - 128);
    tc::fence_async_smem();
    __syncthreads();
    load_kp(c - 1);
#pragma unroll
    for (int x = 0; x < W / 4; ++x) {
      const int i = (tid + 256 * x) / W, j = (tid + 256 * x) % W;
      float val = 0.f;
#pragma unroll
      for (int y = 0; y < SP; ++y) val += partP[(y * W + j) * LD + i];  // (P^T dO lies column by column)
      val = fmaf(s[R + i], slab_sum<W>(part, R, i, j), val);
      Vn[i * W + j] = -val;
      if (i < C && j0 + j < V) p.dvn[(ci * C + i) * V + j0 + j] = val;
    }
    if (tma) ok = tc::mbar_wait(bar + 1, ph);
    ok = __syncthreads_and(ok);  // dv_new, q and w are in place
    if (!ok) break;
    if (tid < 128) slab_tn<W, KP, R>(part, Qs, Od, tid);
    else slab_tn<W, KP, R>(partW, Ws, Vn, tid - 128);
    tc::fence_async_smem();
    __syncthreads();
    load_qw(c - 1);
    slab_state_step<W, KP, 2 * SPK>(St, part, s[2 * R], c > 0 ? p.dhs + (ci - 1) * V * K : nullptr, K, V, p.vecK, j0);
    if (c > 0) put(c - 1);
  }
  if (!ok && tid == 0) atomicExch(p.status, 5);
  if (p.dh0 && ok) {
    __syncthreads();
    slab_state_out<W, KP>(St, p.dh0 + (size_t)bh * K * V, K, V, j0);
  }
}

// ----------------------------------------------------------- chunk backward
// One CTA per chunk, everything that is not the sequential pass.  With e = T^T dv_new and z = T^T dw = -e S0^T
// (dw = -dv_new S0^T is never formed):
//   dPG = tril(dO v_new^T) Gamma                       dq = E(gam) dO S0^T + dPG k
//   Y = e (v beta)^T + z (k beta E(gam))^T             M = -tril(Y T^T, -1) Gamma,  Mb = beta_i M
//   dk = r (v_new dS^T) + dPG^T q + (Mb + Mb^T) k + beta E(gam) z            dv = beta e
//   dbeta = e.v + E(gam) (k.z) + sum_j M_ij (k_i.k_j)
//   dgam_i = q_i.(E(gam) dO S0^T)_i - k_i.(r v_new dS^T)_i + beta_i E(gam_i) (k_i.z_i)
//            + the row sums minus the column sums of (dP P) and of (Mb k k^T), below the diagonal,
//   dgam_last += L <dS,S0> + sum_i r_i k_i.(v_new dS^T)_i
// (The row and column sums are the parts of q.dq and k.dk that come from dPG and Mb, so q.dq - k.dk + 2 (..) needs no sums.
// But it cancels what it need not form: the diagonal of dP P and twice the A terms.  Its dgate was 1.5 to 2.4 times as far
// from a float64 scan, with nothing gained in time.)
// Three 64 x 64 matrices live in shared memory, every wide operand is streamed; e and z make a round trip through the
// workspace (L2).  106 KB: two CTAs per SM.
constexpr int kChunkF32Smem = (simt::kStageFloats + 3 * simt::R * simt::LD + 10 * simt::R + 16) * 4;
static_assert(2 * (kChunkF32Smem + 1024) <= 228 * 1024, "two CTAs per SM");

template <typename IO, int NGK>
__global__ void __launch_bounds__(256, 2) gdn_chunk_bwd_kernel(GdnP p) {
  begin_dependent();
  using namespace simt;
  extern __shared__ __align__(16) float smem[];
  float* stage = smem;
  float* Tm = stage + kStageFloats;  // [64][LD] T
  float* X1 = Tm + R * LD;           // dP Gamma
  float* X2 = X1 + R * LD;           // Y, then Mb + Mb^T
  float* gam = X2 + R * LD;
  float* bet = gam + R;
  float* dd = bet + R;
  float* rr = dd + R;
  float* bd = rr + R;
  float* rs = bd + R;    // row sums of M (k k^T)
  float* dbe = rs + R;   // dbeta
  float* dg = dbe + R;   // dgam
  float* rho = dg + R;   // k_i . dkp_i
  float* pw = rho + R;   // row sums minus column sums of dP P
  float* red = pw + R;   // [8]
  const int C = p.C, K = p.K, V = p.V;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31, warp = tid >> 5;
  const int c = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh % p.H, t0 = c * C;
  const size_t ci = (size_t)bh * p.n + c;
  const int imax = min(C, p.T - t0);
  auto row = [&](int i) { return ((size_t)(b * p.T + t0 + i) * p.H + h); };
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const IO *q = static_cast<const IO*>(p.q), *k = static_cast<const IO*>(p.k);
  const IO *v = static_cast<const IO*>(p.v), *dO = static_cast<const IO*>(p.dO);
  auto ldq = [&](int i, int x) { return i < imax ? ld4(q + row(i) * K, x, K, p.vecK) : zero; };
  auto ldk = [&](int i, int x) { return i < imax ? ld4(k + row(i) * K, x, K, p.vecK) : zero; };
  auto ldv = [&](int i, int x) { return i < imax ? ld4(v + row(i) * V, x, V, p.vecV) : zero; };
  auto ldo = [&](int i, int x) { return i < imax ? ld4(dO + row(i) * V, x, V, p.vecV) : zero; };
  const float *hs = p.hs + ci * V * K, *dhs = p.dhs + ci * V * K;
  const float *vn = p.vn + ci * C * V, *dvn = p.dvn + ci * C * V;
  float *e = p.e + ci * C * V, *z = p.z + ci * C * K;
  auto lde = [&](int i, int x) { return i < C ? ld4(e + i * V, x, V, p.vecV) : zero; };
  auto ldz = [&](int i, int x) { return i < C ? ld4(z + i * K, x, K, p.vecK) : zero; };
  auto ldvn = [&](int i, int x) { return i < C ? ld4(vn + i * V, x, V, p.vecV) : zero; };
  auto lddvn = [&](int i, int x) { return i < C ? ld4(dvn + i * V, x, V, p.vecV) : zero; };
  auto ldhs = [&](int j, int x) { return j < V ? ld4(hs + (size_t)j * K, x, K, p.vecK) : zero; };
  auto lddhs = [&](int j, int x) { return j < V ? ld4(dhs + (size_t)j * K, x, K, p.vecK) : zero; };

  if (tid < R) {
    const float gl = p.gam[ci * C + C - 1], g = tid < C ? p.gam[ci * C + tid] : gl;
    const float bt = tid < imax ? p.beta[row(tid)] : 0.f, d = exp_nonpos_precise(g);
    gam[tid] = g;
    bet[tid] = bt;
    dd[tid] = d;
    rr[tid] = exp_nonpos_precise(gl - g);
    bd[tid] = bt * d;
  }
  for (int u = tid; u < R * R; u += 256) {
    const int i = u >> 6, j = u & 63;
    Tm[i * LD + j] = (i < C && j < C) ? p.Tm[ci * C * C + i * C + j] : 0.f;
  }
  {  // <dS, S0>
    float part = 0.f;
    if (p.vecK) {
      for (int u = 4 * tid; u < V * K; u += 1024)
        part = dot4(*reinterpret_cast<const float4*>(hs + u), *reinterpret_cast<const float4*>(dhs + u), part);
    } else {
      for (int u = tid; u < V * K; u += 256) part = fmaf(hs[u], dhs[u], part);
    }
    part = warp_sum(part);
    if (lane == 0) red[warp] = part;
  }
  // ---- e = T^T dv_new, dv = beta e, e.v ----
  {
    float vd[4] = {0.f, 0.f, 0.f, 0.f};
    IO* dv = static_cast<IO*>(p.dv);
    auto product = [&](auto ng, int j0) {
      constexpr int NG = decltype(ng)::value;
      f2 acc[4][2 * NG];
      clear(acc);
      stream_nn<NG, 2>(acc, stage, R, Tm, NoA{}, [&](int m, int x) { return lddvn(m, j0 + x); });
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          const int i = 4 * ty + r, j = j0 + 64 * g + 4 * tx;
          const float4 x = acc4<NG>(acc, r, g);
          if (i < C) st4(e + i * V, j, V, p.vecV, x);
          if (i < imax) {
            vd[r] = dot4(x, ldv(i, j), vd[r]);
            st4(dv + row(i) * V, j, V, p.vecV, scale4(x, bet[i]));
          }
        }
    };
    if (V <= 64) product(std::integral_constant<int, 1>{}, 0);
    else
      for (int j0 = 0; j0 < V; j0 += 128) product(std::integral_constant<int, 2>{}, j0);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      vd[r] = row_sum(vd[r]);
      if (tx == 0) dbe[4 * ty + r] = vd[r];
    }
  }
  // Column sums of a 64 x 64 result held as rows ty + 16 r, columns tx + 16 x, each thread's four rows added already: the
  // two rows of a warp, then the warps in order, by the first 64 threads.  In the streaming buffers, which are free.
  auto col_sums = [&](const float (&v)[4]) {
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float s = v[x] + __shfl_xor_sync(0xffffffffu, v[x], 16);
      if (lane < 16) stage[warp * R + tx + 16 * x] = s;
    }
    __syncthreads();
    float s = 0.f;
    if (tid < R)
      for (int w = 0; w < 8; ++w) s += stage[w * R + tid];
    return s;
  };
  // ---- dP Gamma, and the sums of dP P ----
  {
    f2 acc[4][4];
    clear(acc);
    stream_nt(acc, stage, V, ldo, ldvn);
    const float* P = p.P + ci * C * C;
    float cs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = ty + 16 * r;
      float sum = 0.f;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int j = tx + 16 * x;
        const float dP = sum2(acc[r][x]);
        X1[i * LD + j] = (i >= j) ? dP * exp_nonpos_precise(gam[i] - gam[j]) : 0.f;
        const float w = (i > j && i < C) ? dP * P[i * C + j] : 0.f;
        sum += w;
        cs[x] += w;
      }
      sum = row_sum(sum);
      if (tx == 0) pw[i] = sum;
    }
    const float col = col_sums(cs);
    if (tid < R) pw[tid] -= col;
  }
  // ---- dq = E(gam) dO S0^T + dPG k ----
  {
    f2 acc[4][2 * NGK];
    clear(acc);
    stream_nn<NGK, 0>(acc, stage, V, nullptr, ldo, ldhs);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const f2 s = pack2(dd[4 * ty + r], dd[4 * ty + r]);
#pragma unroll
      for (int x = 0; x < 2 * NGK; ++x) acc[r][x] = mul2(acc[r][x], s);
      float qd = 0.f;
#pragma unroll
      for (int g = 0; g < NGK; ++g) qd = dot4(acc4<NGK>(acc, r, g), ldq(4 * ty + r, 64 * g + 4 * tx), qd);
      qd = row_sum(qd);
      if (tx == 0) dg[4 * ty + r] = qd;
    }
    stream_nn<NGK, 1>(acc, stage, R, X1, NoA{}, ldk);
    IO* dq = static_cast<IO*>(p.dq);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = 4 * ty + r;
#pragma unroll
      for (int g = 0; g < NGK; ++g)
        if (i < imax) st4(dq + row(i) * K, 64 * g + 4 * tx, K, p.vecK, acc4<NGK>(acc, r, g));
    }
  }
  // ---- z = -e S0^T, k.z ----
  {
    f2 acc[4][2 * NGK];
    clear(acc);
    stream_nn<NGK, 0>(acc, stage, V, nullptr, lde, ldhs);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = 4 * ty + r;
      float kz = 0.f;
#pragma unroll
      for (int g = 0; g < NGK; ++g) {
        const int j = 64 * g + 4 * tx;
        const float4 x = scale4(acc4<NGK>(acc, r, g), -1.f);
        kz = dot4(x, ldk(i, j), kz);
        if (i < C) st4(z + i * K, j, K, p.vecK, x);
      }
      kz = row_sum(kz);
      if (tx == 0) {
        dbe[i] += dd[i] * kz;
        dg[i] += bd[i] * kz;
      }
    }
    __syncthreads();  // e and z are complete
  }
  // ---- Y = e (v beta)^T + z (k beta E(gam))^T, dA = tril(Y T^T, -1), M ----
  {
    f2 acc[4][4];
    clear(acc);
    stream_nt(acc, stage, V, lde, [&](int m, int x) { return scale4(ldv(m, x), bet[m]); });
    stream_nt(acc, stage, K, ldz, [&](int m, int x) { return scale4(ldk(m, x), bd[m]); });
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int x = 0; x < 4; ++x) X2[(ty + 16 * r) * LD + tx + 16 * x] = sum2(acc[r][x]);
    f2 kk[4][4];
    clear(kk);
    stream_nt(kk, stage, K, ldk, ldk);  // its barriers publish Y
    clear(acc);
    tile_nt(acc, X2, LD, Tm, LD, R);
    __syncthreads();  // Y has been read
    float cs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = ty + 16 * r;
      float sum = 0.f;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int j = tx + 16 * x;
        if (i > j) {
          const float M = -sum2(acc[r][x]) * exp_nonpos_precise(gam[i] - gam[j]), w = M * sum2(kk[r][x]);
          sum += w;
          cs[x] = fmaf(bet[i], w, cs[x]);
          X2[i * LD + j] = bet[i] * M;
          X2[j * LD + i] = bet[i] * M;
        } else if (i == j) {
          X2[i * LD + i] = 0.f;
        }
      }
      sum = row_sum(sum);
      if (tx == 0) rs[i] = sum;
    }
    const float col = col_sums(cs);
    if (tid < R) pw[tid] -= col;
  }
  // ---- dk ----
  {
    f2 acc[4][2 * NGK];
    clear(acc);
    stream_nn<NGK, 0>(acc, stage, V, nullptr, ldvn, lddhs);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = 4 * ty + r;
      const f2 s = pack2(rr[i], rr[i]);
      float kp = 0.f;
#pragma unroll
      for (int g = 0; g < NGK; ++g) {
        acc[r][2 * g] = mul2(acc[r][2 * g], s);
        acc[r][2 * g + 1] = mul2(acc[r][2 * g + 1], s);
        kp = dot4(acc4<NGK>(acc, r, g), ldk(i, 64 * g + 4 * tx), kp);
      }
      kp = row_sum(kp);
      if (tx == 0) rho[i] = kp;
    }
    stream_nn<NGK, 2>(acc, stage, R, X1, NoA{}, ldq);
    stream_nn<NGK, 1>(acc, stage, R, X2, NoA{}, ldk);
    IO* dk = static_cast<IO*>(p.dk);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = 4 * ty + r;
#pragma unroll
      for (int g = 0; g < NGK; ++g) {
        const int j = 64 * g + 4 * tx;
        const float4 a = acc4<NGK>(acc, r, g), zz = ldz(i, j);
        const float4 x = make_float4(fmaf(bd[i], zz.x, a.x), fmaf(bd[i], zz.y, a.y), fmaf(bd[i], zz.z, a.z), fmaf(bd[i], zz.w, a.w));
        if (i < imax) st4(dk + row(i) * K, j, K, p.vecK, x);
      }
      if (tx == 0) {
        dbe[i] += rs[i];
        dg[i] += pw[i] + bet[i] * rs[i] - rho[i];
      }
    }
  }
  __syncthreads();
  if (tid < 32) {  // dg = reverse cumulative sum of dgam within the chunk: one warp, two rows per lane
    float base = 0.f;
    for (int x = 0; x < 8; ++x) base += red[x];
    base = exp_nonpos_precise(gam[R - 1]) * base + warp_sum(rho[tid] + rho[tid + 32]);
    const int ra = R - 1 - 2 * tid, rb = ra - 1;
    float a = dg[ra], bq = dg[rb];
    warp_rcumsum64(a, bq, tid);
    __syncwarp();
    dg[ra] = base + a;
    dg[rb] = base + bq;
  }
  __syncthreads();
  if (tid < imax) {
    p.dbeta[row(tid)] = dbe[tid];
    float x = dg[tid];
    const float gin = p.gate[row(tid)];
    if (p.gate_is_log) {
      if (gin < kLogGateFloor) x = 0.f;
    } else {
      x = (gin > kGateFloor) ? x / gin : 0.f;
    }
    p.dgate[row(tid)] = x;
  }
}

// --------------------------------------------------- token-by-token forward
template <typename IO>
__global__ void __launch_bounds__(256) gdn_recurrent_fwd_kernel(GdnP p) {
  begin_dependent();
  extern __shared__ float smem[];
  const int K = p.K, V = p.V;
  float* S = smem;           // [K][33]
  float* sk = S + K * 33;    // [K]
  float* sq = sk + K;        // [K]
  float* red = sq + K;       // [2][8][32]
  const int tid = threadIdx.x, j = tid & 31, rg = tid >> 5;
  const int bh = blockIdx.y, b = bh / p.H, h = bh % p.H;
  const int jv = blockIdx.x * 32 + j;
  const bool jok = jv < V;
  const IO* q = static_cast<const IO*>(p.q);
  const IO* k = static_cast<const IO*>(p.k);
  const IO* v = static_cast<const IO*>(p.v);
  IO* out = static_cast<IO*>(p.out);
  for (int kk = rg; kk < K; kk += 8)
    S[kk * 33 + j] = (p.h0 && jok) ? p.h0[((size_t)bh * K + kk) * V + jv] : 0.f;
  for (int t = 0; t < p.T; ++t) {
    const size_t r = (size_t)(b * p.T + t) * p.H + h;
    __syncthreads();
    for (int i = tid; i < K; i += blockDim.x) {
      sk[i] = to_f32(k[r * K + i]);
      sq[i] = to_f32(q[r * K + i]);
    }
    __syncthreads();
    const float gv = p.gate[r];
    const float a = p.gate_is_log ? expf(gv) : gv;
    float pk = 0.f, pq = 0.f, qk = 0.f;
    for (int kk = rg; kk < K; kk += 8) {
      const float s = S[kk * 33 + j];
      pk = fmaf(sk[kk], s, pk);
      pq = fmaf(sq[kk], s, pq);
    }
    for (int kk = 0; kk < K; ++kk) qk = fmaf(sq[kk], sk[kk], qk);
    red[rg * 32 + j] = pk;
    red[256 + rg * 32 + j] = pq;
    __syncthreads();
    pk = 0.f; pq = 0.f;
    for (int wv = 0; wv < 8; ++wv) { pk += red[wv * 32 + j]; pq += red[256 + wv * 32 + j]; }
    const float vv = jok ? to_f32(v[r * V + jv]) : 0.f;
    const float e = p.beta[r] * (vv - a * pk);
    for (int kk = rg; kk < K; kk += 8) S[kk * 33 + j] = fmaf(sk[kk], e, a * S[kk * 33 + j]);
    if (rg == 0 && jok) out[r * V + jv] = from_f32<IO>(fmaf(qk, e, a * pq));
  }
  __syncthreads();
  if (p.hT && jok)
    for (int kk = rg; kk < K; kk += 8) p.hT[((size_t)bh * K + kk) * V + jv] = S[kk * 33 + j];
}

// ------------------------------------------------------------------ host
static size_t carve(GdnP& p, void* ws, bool bwd) {
  Carver cv(ws);
  const size_t nc = (size_t)p.B * p.H * p.n, C = p.C, K = p.K, V = p.V;
  p.status = cv.take<int>(64);
  p.gam = cv.take<float>(nc * C);
  p.Tm = cv.take<float>(nc * C * C);
  p.w = cv.take<float>(nc * C * K);
  p.u = cv.take<float>(nc * C * V);
  p.P = cv.take<float>(nc * C * C);
  if (bwd) {
    p.hs = cv.take<float>(nc * V * K);
    p.vn = cv.take<float>(nc * C * V);
    p.dhs = cv.take<float>(nc * V * K);
    p.dvn = cv.take<float>(nc * C * V);
    p.e = cv.take<float>(nc * C * V);
    p.z = cv.take<float>(nc * C * K);
  }
  return cv.bytes();
}

static GdnP make_params(const mxb_gdn_desc* d) {
  GdnP p{};
  p.B = d->B; p.T = d->T; p.H = d->H; p.K = d->Dk; p.V = d->Dv;
  p.C = d->chunk > 64 ? 64 : d->chunk;
  if (p.C < 2) p.C = 64;  // the backward of the token recurrence runs in chunked form
  p.n = (d->T + p.C - 1) / p.C;
  p.gate_is_log = d->gate_is_log;
  return p;
}

size_t gdn_simt_workspace_bytes(const mxb_gdn_desc* d, bool bwd) {
  if (!bwd && d->chunk <= 1) return 0;
  GdnP p = make_params(d);
  return carve(p, nullptr, bwd);
}

// Any chunk size is accepted: the result does not depend on it, and sizes above 64 are computed
// with chunks of 64 (make_params), as the reference allows larger scan_chunk_size overrides
// (arch/blocks_gated_deltanet.go:11-17).  Dv up to 256 covers the reference default Dv = 2 Dk.
bool gdn_simt_supported(const mxb_gdn_desc* d) {
  return d->Dk >= 1 && d->Dv >= 1 && d->Dk <= 128 && d->Dv <= 256;
}

// Rows can be moved four elements at a time where the width is a multiple of four and every tensor of that width is
// aligned to four elements (the workspace always is).
template <typename IO>
static bool vec_ok(int width, std::initializer_list<const void*> tensors) {
  uintptr_t bits = 0;
  for (const void* t : tensors) bits |= reinterpret_cast<uintptr_t>(t);
  return width % 4 == 0 && bits % (4 * sizeof(IO)) == 0;
}

template <typename IO, int KP>
static mxb_status run_prep(GdnP p, cudaStream_t st) {
  SlabMaps maps;
  std::memset(&maps, 0, sizeof maps);
  p.tma = sizeof(IO) == 4 && p.C == simt::R && make_tma_map_f32(&maps.q, p.q, p.B, p.T, p.H, p.K) &&
          make_tma_map_f32(&maps.k, p.k, p.B, p.T, p.H, p.K);
  p.vtma = sizeof(IO) == 4 && p.C == simt::R && make_tma_map_f32(&maps.P, p.v, p.B, p.T, p.H, p.V);
  constexpr int sm = PrepF32<KP>::smem;
  if (MXB_ALLOW_SMEM(sm, gdn_prep_kernel<IO, KP>) != MXB_OK) return MXB_ERR_CUDA;
  MXB_LAUNCH("gdn_prep_kernel", st, (launch_kernel(gdn_prep_kernel<IO, KP>, dim3(p.n, p.B * p.H), 256, sm, st, p, maps)));
  return check_launch("gdn_prep_kernel");
}

// Columns of a state CTA: the narrowest slab whose CTAs are on the 148 SMs at once (a chunk takes less time the narrower
// the slab is), 16 where even those come in several rounds: per column the wide slab is the cheapest.
static int slab_columns(const GdnP& p) {
  for (int w = 4; w < 16; w *= 2)
    if ((size_t)p.B * p.H * ((p.V + w - 1) / w) <= 148) return w;
  return 16;
}
template <typename IO, int W, int KP>
static mxb_status run_state(GdnP p, bool bwd, cudaStream_t st) {
  SlabMaps maps;
  std::memset(&maps, 0, sizeof maps);
  const int rows = p.B * p.H * p.n * p.C;
  p.tma = sizeof(IO) == 4 && p.C == simt::R && make_tma_map_f32(&maps.q, p.q, p.B, p.T, p.H, p.K) &&
          make_tma_map_f32(&maps.k, p.k, p.B, p.T, p.H, p.K) && make_tma_map_f32(&maps.w, p.w, 1, rows, 1, p.K) &&
          make_tma_map_f32(&maps.P, p.P, 1, rows, 1, simt::R);
  const dim3 grid((p.V + W - 1) / W, p.B * p.H);
  if (bwd) {
    constexpr int sm = state_bwd_smem<W, KP>();
    if (MXB_ALLOW_SMEM(sm, gdn_state_bwd_kernel<IO, W, KP>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_state_bwd_kernel", st, (launch_kernel(gdn_state_bwd_kernel<IO, W, KP>, grid, 256, sm, st, p, maps)));
    return check_launch("gdn_state_bwd_kernel");
  }
  constexpr int sm = state_fwd_smem<W, KP>();
  if (MXB_ALLOW_SMEM(sm, gdn_state_fwd_kernel<IO, W, KP>) != MXB_OK) return MXB_ERR_CUDA;
  MXB_LAUNCH("gdn_state_fwd_kernel", st, (launch_kernel(gdn_state_fwd_kernel<IO, W, KP>, grid, 256, sm, st, p, maps)));
  return check_launch("gdn_state_fwd_kernel");
}
template <typename IO>
static mxb_status run_state(const GdnP& p, bool bwd, cudaStream_t st) {
  const bool narrow = p.K <= 64;
  switch (slab_columns(p)) {
    case 4: return narrow ? run_state<IO, 4, 64>(p, bwd, st) : run_state<IO, 4, 128>(p, bwd, st);
    case 8: return narrow ? run_state<IO, 8, 64>(p, bwd, st) : run_state<IO, 8, 128>(p, bwd, st);
    default: return narrow ? run_state<IO, 16, 64>(p, bwd, st) : run_state<IO, 16, 128>(p, bwd, st);
  }
}
template <typename IO, int NGK>
static mxb_status run_chunk_bwd(const GdnP& p, cudaStream_t st) {
  if (MXB_ALLOW_SMEM(kChunkF32Smem, gdn_chunk_bwd_kernel<IO, NGK>) != MXB_OK) return MXB_ERR_CUDA;
  MXB_LAUNCH("gdn_chunk_bwd_kernel", st,
             (launch_kernel(gdn_chunk_bwd_kernel<IO, NGK>, dim3(p.n, p.B * p.H), 256, kChunkF32Smem, st, p)));
  return check_launch("gdn_chunk_bwd_kernel");
}

template <typename IO>
static mxb_status run_fwd(GdnP& p, bool chunked, cudaStream_t st) {
  const int K = p.K, V = p.V;
  if (!chunked) {
    dim3 gslab((V + 31) / 32, p.B * p.H);
    size_t sm = sizeof(float) * (K * 33 + 2 * K + 512);
    if (MXB_ALLOW_SMEM((int)sm, gdn_recurrent_fwd_kernel<IO>) != MXB_OK) return MXB_ERR_CUDA;
    MXB_LAUNCH("gdn_recurrent_fwd_kernel", st, (launch_kernel(gdn_recurrent_fwd_kernel<IO>, gslab, 256, sm, st, p)));
    return check_launch("gdn_recurrent_fwd_kernel");
  }
  p.vecK = vec_ok<IO>(K, {p.q, p.k, p.dq, p.dk});
  p.vecV = vec_ok<IO>(V, {p.v, p.dO, p.dv});
  mxb_status s = K <= 64 ? run_prep<IO, 64>(p, st) : run_prep<IO, 128>(p, st);
  if (s != MXB_OK) return s;
  return run_state<IO>(p, false, st);
}

template <typename IO>
static mxb_status run_bwd(GdnP& p, bool recompute, cudaStream_t st) {
  const int K = p.K, V = p.V;
  p.save = 1;
  mxb_status s = MXB_OK;
  if (recompute) {
    // forward recompute into the workspace; out is not needed -> write into dv (overwritten later)
    void* keep_out = p.out;
    float* keep_hT = p.hT;
    p.out = p.dv;
    p.hT = nullptr;
    s = run_fwd<IO>(p, true, st);
    p.out = keep_out;
    p.hT = keep_hT;
    if (s != MXB_OK) return s;
  }
  p.vecK = vec_ok<IO>(K, {p.q, p.k, p.dq, p.dk});
  p.vecV = vec_ok<IO>(V, {p.v, p.dO, p.dv});
  s = run_state<IO>(p, true, st);
  if (s != MXB_OK) return s;
  return K <= 64 ? run_chunk_bwd<IO, 1>(p, st) : run_chunk_bwd<IO, 2>(p, st);
}

mxb_status gdn_simt_fwd(const mxb_gdn_desc* d, const void* q, const void* k, const void* v,
                        const float* beta, const float* gate, const float* h0, void* out, float* hT,
                        void* ws, cudaStream_t st) {
  GdnP p = make_params(d);
  p.q = q; p.k = k; p.v = v; p.beta = beta; p.gate = gate; p.h0 = h0; p.out = out; p.hT = hT;
  const bool chunked = d->chunk > 1;
  if (chunked) {
    p.save = (d->flags & MXB_GDN_SAVE_FOR_BWD) ? 1 : 0;
    carve(p, ws, p.save != 0);
  }
  return d->io_dtype == MXB_F32 ? run_fwd<float>(p, chunked, st) : run_fwd<__nv_bfloat16>(p, chunked, st);
}

mxb_status gdn_simt_bwd(const mxb_gdn_desc* d, const void* q, const void* k, const void* v,
                        const float* beta, const float* gate, const float* h0, const void* dO,
                        const float* dhT, void* dq, void* dk, void* dv, float* dbeta, float* dgate,
                        float* dh0, void* ws, cudaStream_t st) {
  GdnP p = make_params(d);
  p.q = q; p.k = k; p.v = v; p.beta = beta; p.gate = gate; p.h0 = h0;
  p.dO = dO; p.dhT_in = dhT; p.dq = dq; p.dk = dk; p.dv = dv; p.dbeta = dbeta; p.dgate = dgate; p.dh0 = dh0;
  carve(p, ws, true);
  // saved intermediates exist only for the chunked forward
  const bool recompute = !(d->flags & MXB_GDN_BWD_USE_SAVED) || d->chunk <= 1;
  return d->io_dtype == MXB_F32 ? run_bwd<float>(p, recompute, st) : run_bwd<__nv_bfloat16>(p, recompute, st);
}

}  // namespace mxb
