// Mixture head of one row from its raw outputs: what the fp32 dense kernels share.
#pragma once
#include "dense.cuh"

namespace artab {

// One warp per head row: mixture parameters from raw[3K], then sample or log-pdf.
__device__ __forceinline__ void head_row(const DenseArgs& a, const float* raw, long row) {
  const int lane = threadIdx.x & 31;
  const int K = a.n_comp;
  const long b = row / a.head_tps;
  const int j = (int)(row - b * a.head_tps);
  if (j < a.head_first) return;
  const long oidx = b * a.out_stride + a.out_col + (j - a.head_first);
  float mean = 0.f, stdv = 1.f, lw = -INFINITY;
  if (lane < K) {
    mean = raw[3 * lane] + __ldg(a.mean_bias + lane);
    const float sr = raw[3 * lane + 1] + __ldg(a.std_bias + lane);
    const float sp = sr > 20.f ? sr : log1pf(expf(sr));  // F.softplus, beta 1, threshold 20
    stdv = fminf(sp, 2.0f) + 1e-3f;
    lw = raw[3 * lane + 2] + __ldg(a.weight_bias + lane);
  }
  const float mx = warp_max(lw);
  const float se = warp_sum(lane < K ? expf(lw - mx) : 0.f);
  const float logw = lw - mx - logf(se);  // log_softmax
  float y;
  if (a.head_mode == 1) {
    // torch.multinomial(w, 1) == argmax_k(w_k / Exp(1)_k); first maximum wins
    float ratio = -1.f;
    if (lane < K) ratio = expf(logw) / __ldg(a.expo + b * K + lane);
    int best = lane;
    float bv = ratio;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best, o);
      if (ov > bv || (ov == bv && oi < best)) {
        bv = ov;
        best = oi;
      }
    }
    const float m_sel = __shfl_sync(0xffffffffu, mean, best);
    const float s_sel = __shfl_sync(0xffffffffu, stdv, best);
    y = m_sel + s_sel * __ldg(a.normal + b);
    if (lane == 0) {
      a.y_out[oidx] = y;
      if (a.comp_out) a.comp_out[oidx] = best;
    }
  } else {
    y = __ldg(a.y_in + oidx);
  }
  if (a.ld_out) {
    float lp = -INFINITY;
    if (lane < K) {
      const float zz = (y - mean) / stdv;
      lp = -0.5f * (1.8378770664093453f + 2.0f * logf(stdv) + zz * zz) + logw;
    }
    const float m2 = warp_max(lp);
    const float s2 = warp_sum(lane < K ? expf(lp - m2) : 0.f);
    if (lane == 0) a.ld_out[oidx] = m2 + logf(s2);
  }
}

}  // namespace artab
