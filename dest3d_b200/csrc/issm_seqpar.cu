// Support for cutting one sequence into slices (over several GPUs, or as extra batch entries on one): the decay a
// slice applies to the state entering it is exp(A * sum of the transformed step sizes of the slice), the role the
// per-chunk `dA_cumsum[..., -1]` plays in the reference's state passing (issm_triton/issm_state_passing.py:92-107).
// This kernel produces the sums; one read of dt, coalesced over the states.
#include "issm_common.cuh"

namespace issm {

// part[seg, b, h, n] = sum over the rows of segment `seg` of clamp(softplus?(dt[b, l, h, n] + bias[h, n]))
template <typename T>
__global__ void __launch_bounds__(256) k_dt_sum(const T* __restrict__ dt, int64_t sb, int64_t sl, int64_t sh, const float* __restrict__ bias,
                                                 int softplus, float lo, float hi, int L, int rows, int N, float* __restrict__ part) {
  const int seg = blockIdx.x, h = blockIdx.y, b = blockIdx.z, H = gridDim.y, Bn = gridDim.z;
  const int l0 = seg * rows, l1 = min(L, l0 + rows);
  const T* p = dt + b * sb + h * sh;
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    const float bv = bias ? bias[h * N + n] : 0.f;
    float acc = 0.f;
#pragma unroll 8
    for (int l = l0; l < l1; ++l) {
      float v = ldf(p + (int64_t)l * sl + n) + bv;
      if (softplus) v = softplus_thr(v);
      acc += fminf(fmaxf(v, lo), hi);
    }
    part[(((size_t)seg * Bn + b) * H + h) * N + n] = acc;
  }
}
}  // namespace issm

using namespace issm;

extern "C" int issm_b200_dt_sum(const void* dt, int32_t dt_dtype, int32_t batch, int32_t seqlen, int32_t nheads, int32_t dstate,
                                int64_t dt_sb, int64_t dt_sl, int64_t dt_sh, const float* dt_bias, int32_t dt_softplus, float dt_min,
                                float dt_max, int32_t rows_per_part, float* part, void* stream) {
  if (!dt || !part) return ISSM_ERR_NULL;
  if (batch <= 0 || batch > 65535 || seqlen <= 0 || nheads <= 0 || nheads > 65535 || dstate <= 0 || rows_per_part <= 0) return ISSM_ERR_SHAPE;
  if (dt_dtype != ISSM_F32 && dt_dtype != ISSM_BF16) return ISSM_ERR_DTYPE;
  const dim3 grid((seqlen + rows_per_part - 1) / rows_per_part, nheads, batch);
  const int threads = dstate >= 256 ? 256 : ((dstate + 31) / 32) * 32;
  cudaStream_t s = (cudaStream_t)stream;
  if (dt_dtype == ISSM_F32)
    ISSM_LAUNCH(k_dt_sum<float>, grid, threads, 0, s, (const float*)dt, dt_sb, dt_sl, dt_sh, dt_bias, dt_softplus, dt_min, dt_max, seqlen, rows_per_part, dstate, part);
  else
    ISSM_LAUNCH(k_dt_sum<bf16>, grid, threads, 0, s, (const bf16*)dt, dt_sb, dt_sl, dt_sh, dt_bias, dt_softplus, dt_min, dt_max, seqlen, rows_per_part, dstate, part);
  return ISSM_OK;
}

// One thread per (sequence, head, channel, state) walks the slices: run = F + 2^sums run, coalesced over the states.
namespace issm {
__global__ void k_slice_chain(const __grid_constant__ issm_slice_chain q) {
  const int64_t hpn = (int64_t)q.nheads * q.headdim * q.dstate, i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= q.batch * hpn) return;
  const int64_t b = i / hpn, e = i - b * hpn;
  const int n = (int)(e % q.dstate), h = (int)(e / ((int64_t)q.headdim * q.dstate));
  const int64_t hn = (int64_t)q.nheads * q.dstate, sn = (int64_t)h * q.dstate + n;
  const int total = q.nmain + (q.f_tail ? 1 : 0);
  float run = !q.start ? 0.f : q.start_f32 ? ((const float*)q.start)[i] : ldf((const bf16*)q.start + i);
  for (int k0 = 0; k0 < total; k0 += 8) {                  // eight slices' loads at once: one latency, not eight
    float local[8], sum[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int c = min(k0 + k, total - 1), s = q.descending ? total - 1 - c : c;
      const bool tail = s == q.nmain;
      const int64_t row = tail ? b : b * q.nmain + s;
      local[k] = (tail ? q.f_tail : q.f_main)[row * hpn + e];
      sum[k] = (tail ? q.s_tail : q.s_main)[row * hn + sn];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (k0 + k >= total) break;
      const int s = q.descending ? total - 1 - k0 - k : k0 + k;
      const bool tail = s == q.nmain;
      const int64_t at = (tail ? b : b * q.nmain + s) * hpn + e;
      void* en = tail ? q.enter_tail : q.enter_main;
      if (q.enter_f32) ((float*)en)[at] = run;
      else stf((bf16*)en + at, run);
      run = fmaf(exp2f(sum[k]), run, local[k]);
    }
  }
  if (q.last) {
    if (q.last_f32) ((float*)q.last)[i] = run;
    else stf((bf16*)q.last + i, run);
  }
}
}  // namespace issm

extern "C" size_t issm_b200_sizeof_slice_chain(void) { return sizeof(issm_slice_chain); }
extern "C" int issm_b200_slice_chain(const issm_slice_chain* p, void* stream) {
  if (!p || !p->f_main || !p->s_main || !p->enter_main || (p->f_tail && (!p->s_tail || !p->enter_tail))) return ISSM_ERR_NULL;
  if (p->batch <= 0 || p->nmain <= 0 || p->nheads <= 0 || p->headdim <= 0 || p->dstate <= 0) return ISSM_ERR_SHAPE;
  const int64_t n = (int64_t)p->batch * p->nheads * p->headdim * p->dstate;
  ISSM_LAUNCH(k_slice_chain, (unsigned)cdiv64(n, 128), 128, 0, (cudaStream_t)stream, *p);
  return ISSM_OK;
}
