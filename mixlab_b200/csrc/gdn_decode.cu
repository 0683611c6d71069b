// Gated delta rule - single-token recurrent decode step (HBM-bound stream).
//
// Semantics: the loop body of the reference's gated_delta_scan_naive
// (gpu/ir.cpp:2334-2345) applied once to a persistent fp32 state [N,H,Dk,Dv]:
//     S <- a S ; pred = k^T S ; S <- S + k (x) beta (v - pred) ; o = q^T S
//
// The state is read once and written once.  Both contractions over Dk are taken
// from the SAME pass over the loaded state:
//     pred = a (k^T S_old)         o = a (q^T S_old) + (q.k) beta (v - pred)
// so there is a single cross-warp reduction between the load and the store.
//
// Mapping: the columns of a state are independent, so a CTA of 128 threads takes 32 of them: lane = 4 columns
// (a row of the slab is one 128-byte line, a warp reads four rows with 128-bit loads), thread group rg = tid / 8
// owns rows rg, rg + 16, ... and keeps its ROWS float4 pieces of the state in registers between load and store.
// Many small CTAs keep more loads in flight than a pipeline over shared memory did (64 KB tiles, one persistent CTA per
// SM, bulk copies): a step of 256 sequences x 16 heads of 128 x 128 takes 84 us instead of 95 (6.5 TB/s read + written),
// one sequence 4.1 us beside other steps instead of 17 (most of that was host work).  Bound: HBM, and the launch and the
// latency of one load -> sum -> store chain for the small calls.
#include "common.cuh"

namespace mxb {

template <typename IO, int ROWS>
__global__ void __launch_bounds__(128)
gdn_decode_kernel(float* __restrict__ state, const IO* __restrict__ q, const IO* __restrict__ k,
                  const IO* __restrict__ v, const float* __restrict__ beta,
                  const float* __restrict__ gate, IO* __restrict__ out, int Dk, int Dv,
                  int gate_is_log) {
  begin_dependent();
  __shared__ float s_k[16 * ROWS], s_q[16 * ROWS];
  __shared__ __align__(16) float4 s_red[4][2][8];
  __shared__ float s_qk[4];

  const int tid = threadIdx.x, cg = tid & 7, rg = tid >> 3, lane = tid & 31, warp = tid >> 5;
  const int slabs = (Dv + 31) / 32;
  const size_t sh = blockIdx.x / slabs;
  const int c0 = (blockIdx.x % slabs) * 32 + 4 * cg;
  const bool col_ok = c0 < Dv;

  float* sp = state + sh * Dk * Dv + c0;
  float4 S[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int row = rg + 16 * r;
    S[r] = (col_ok && row < Dk) ? __ldcs(reinterpret_cast<const float4*>(sp + (size_t)row * Dv)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int i = tid; i < 16 * ROWS; i += 128) {
    s_k[i] = i < Dk ? to_f32(k[sh * Dk + i]) : 0.0f;
    s_q[i] = i < Dk ? to_f32(q[sh * Dk + i]) : 0.0f;
  }
  const float gv = gate[sh];
  const float bt = beta[sh];
  float4 vv = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col_ok) {
    const IO* vp = v + sh * Dv + c0;
    vv = make_float4(to_f32(vp[0]), to_f32(vp[1]), to_f32(vp[2]), to_f32(vp[3]));
  }
  const float a = gate_is_log ? expf(gv) : gv;
  __syncthreads();

  float4 pk = make_float4(0.f, 0.f, 0.f, 0.f), pq = pk;
  float qk = 0.f;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const float kr = s_k[rg + 16 * r], qr = s_q[rg + 16 * r];
    pk.x = fmaf(kr, S[r].x, pk.x); pk.y = fmaf(kr, S[r].y, pk.y);
    pk.z = fmaf(kr, S[r].z, pk.z); pk.w = fmaf(kr, S[r].w, pk.w);
    pq.x = fmaf(qr, S[r].x, pq.x); pq.y = fmaf(qr, S[r].y, pq.y);
    pq.z = fmaf(qr, S[r].z, pq.z); pq.w = fmaf(qr, S[r].w, pq.w);
    qk = fmaf(qr, kr, qk);
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) {  // the four row groups of a warp
    pk.x += __shfl_xor_sync(0xffffffffu, pk.x, o); pk.y += __shfl_xor_sync(0xffffffffu, pk.y, o);
    pk.z += __shfl_xor_sync(0xffffffffu, pk.z, o); pk.w += __shfl_xor_sync(0xffffffffu, pk.w, o);
    pq.x += __shfl_xor_sync(0xffffffffu, pq.x, o); pq.y += __shfl_xor_sync(0xffffffffu, pq.y, o);
    pq.z += __shfl_xor_sync(0xffffffffu, pq.z, o); pq.w += __shfl_xor_sync(0xffffffffu, pq.w, o);
    qk += __shfl_xor_sync(0xffffffffu, qk, o);
  }
  if (lane < 8) {
    s_red[warp][0][cg] = pk;
    s_red[warp][1][cg] = pq;
    if (lane == 0) s_qk[warp] = qk;
  }
  __syncthreads();
  pk = s_red[0][0][cg]; pq = s_red[0][1][cg]; qk = s_qk[0];
#pragma unroll
  for (int w = 1; w < 4; ++w) {
    const float4 x = s_red[w][0][cg], y = s_red[w][1][cg];
    pk.x += x.x; pk.y += x.y; pk.z += x.z; pk.w += x.w;
    pq.x += y.x; pq.y += y.y; pq.z += y.z; pq.w += y.w;
    qk += s_qk[w];
  }
  if (!col_ok) return;
  float4 e;
  e.x = bt * (vv.x - a * pk.x); e.y = bt * (vv.y - a * pk.y);
  e.z = bt * (vv.z - a * pk.z); e.w = bt * (vv.w - a * pk.w);
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    const int row = rg + 16 * r;
    if (row < Dk) {
      const float kr = s_k[row];
      float4 n;
      n.x = fmaf(kr, e.x, a * S[r].x); n.y = fmaf(kr, e.y, a * S[r].y);
      n.z = fmaf(kr, e.z, a * S[r].z); n.w = fmaf(kr, e.w, a * S[r].w);
      __stcs(reinterpret_cast<float4*>(sp + (size_t)row * Dv), n);
    }
  }
  if (rg == 0) {
    IO* op = out + sh * Dv + c0;
    op[0] = from_f32<IO>(fmaf(qk, e.x, a * pq.x));
    op[1] = from_f32<IO>(fmaf(qk, e.y, a * pq.y));
    op[2] = from_f32<IO>(fmaf(qk, e.z, a * pq.z));
    op[3] = from_f32<IO>(fmaf(qk, e.w, a * pq.w));
  }
}

template <typename IO>
static mxb_status launch_decode(const mxb_gdn_desc* d, float* state, const void* q, const void* k,
                                const void* v, const float* beta, const float* gate, void* out,
                                cudaStream_t st) {
  const int grid = (d->Dv + 31) / 32 * d->B * d->H;
  auto Q = static_cast<const IO*>(q);
  auto K = static_cast<const IO*>(k);
  auto V = static_cast<const IO*>(v);
  auto O = static_cast<IO*>(out);
  if (d->Dk <= 64)
    MXB_LAUNCH("gdn_decode_kernel", st, (launch_kernel(gdn_decode_kernel<IO, 4>, grid, 128, 0, st, state, Q, K, V, beta, gate, O, d->Dk, d->Dv, d->gate_is_log)));
  else if (d->Dk <= 128)
    MXB_LAUNCH("gdn_decode_kernel", st, (launch_kernel(gdn_decode_kernel<IO, 8>, grid, 128, 0, st, state, Q, K, V, beta, gate, O, d->Dk, d->Dv, d->gate_is_log)));
  else
    MXB_LAUNCH("gdn_decode_kernel", st, (launch_kernel(gdn_decode_kernel<IO, 16>, grid, 128, 0, st, state, Q, K, V, beta, gate, O, d->Dk, d->Dv, d->gate_is_log)));
  return check_launch("gdn_decode_kernel");
}

mxb_status gdn_decode_dispatch(const mxb_gdn_desc* d, float* state, const void* q, const void* k,
                               const void* v, const float* beta, const float* gate, void* out,
                               cudaStream_t st) {
  if (d->Dv % 4 != 0 || d->Dk > 256) return MXB_ERR_UNSUPPORTED;
  if (d->io_dtype == MXB_F32) return launch_decode<float>(d, state, q, k, v, beta, gate, out, st);
  return launch_decode<__nv_bfloat16>(d, state, q, k, v, beta, gate, out, st);
}

}  // namespace mxb
