// pf_obs_terms.cuh -- differenced and carrier-phase observation terms of the
// device filter, one pass over a filter's current particles:
//
//   PF_OBS_DD_PSEUDORANGE  r = dd - (|p - s_k| - |p - s_ref| - b_k + b_ref)   (pf_device.cu:282-368)
//   PF_OBS_CARRIER_AFV     a = afv(cp - (|p - s| + cb) / lambda)              (pf_device.cu:439-494)
//   PF_OBS_DD_CARRIER_AFV  a = afv(dd - (|p - s_k| - |p - s_ref| - b_k + b_ref) / lambda_k)
//                                                                             (pf_device.cu:496-604)
// with afv(v) = v - rint(v), a term -w r^2 / (2 sigma^2) (or the Huber cost
// when huber_k > 0) per row, and for the DD kinds the per-particle gate:
// rows with |r| > gate are dropped unless fewer than min(n, 3) would remain.
//
// Carrier terms resolve centimetres out of 2e7 m ranges, so this kernel
// works in FP64 (the FP32 offsets are exact in FP64).  The rows arrive as a
// kernel parameter in ECEF; every CTA takes them to the filter's local frame
// about its anchor and folds each row's constant part:
//   DD pseudorange    c = dd + b_k - b_ref,               r = c - (r_k - r_ref)
//   carrier           c = cp - clk_anchor / lambda,       a = afv(c - (r + x_clk) / lambda)
//   DD carrier        c = dd + (b_k - b_ref) / lambda_k,  a = afv(c - (r_k - r_ref) / lambda_k)
#pragma once
#include "pf_engine_kernels.cuh"

namespace pfb {

constexpr int kMaxObsRows = 128;

struct ObsRow {
  double sk[3];   // satellite (k) in the local frame
  double sr[3];   // reference satellite in the local frame (DD kinds)
  double c;       // constant part of the residual
  double inv_wl;  // 1 / wavelength (carrier kinds), 1 otherwise
  double w;       // row weight
  double same;    // nonzero: the reference satellite is the previous row's
};

// The caller's rows as a kernel parameter: 32 of them are under the classic
// 4 KB of parameters, sets above that take the larger one.
constexpr int kObsRowsSmall = 32;
template <int CAP>
struct ObsRowsIn {
  pf_obs_row_t row[CAP];
};

struct ObsBlock {
  int n;
  int accumulate;   // 1: add to the current log-weights, 0: overwrite them
  int gate_min;     // rows that must stay inside the gate
  double inv_sigma2;
  double inv_sigma;
  double gate;      // 0: no gate
  double huber_k;   // 0: Gaussian
};

// A row in the filter's local frame, every product and sum rounded by itself.
template <int KIND>
__device__ __forceinline__ ObsRow obs_row(const FilterDesc* fd, const FilterCtrl* fc, const pf_obs_row_t& r,
                                          const pf_obs_row_t* prev) {
  constexpr bool dd = KIND != PF_OBS_CARRIER_AFV;
  ObsRow o;
  double vk[3], vr[3];
  for (int j = 0; j < 3; ++j) {
    vk[j] = __dsub_rn(r.sat_k[j], fc->anchor[j]);
    vr[j] = dd ? __dsub_rn(r.sat_ref[j], fc->anchor[j]) : 0.0;
  }
  for (int q = 0; q < 3; ++q) {
    const double* m = fd->rot + 3 * q;
    o.sk[q] = __dadd_rn(__dadd_rn(__dmul_rn(m[0], vk[0]), __dmul_rn(m[1], vk[1])), __dmul_rn(m[2], vk[2]));
    o.sr[q] = __dadd_rn(__dadd_rn(__dmul_rn(m[0], vr[0]), __dmul_rn(m[1], vr[1])), __dmul_rn(m[2], vr[2]));
  }
  o.w = r.weight;
  o.inv_wl = KIND == PF_OBS_DD_PSEUDORANGE ? 1.0 : 1.0 / r.wavelength;
  if (KIND == PF_OBS_DD_PSEUDORANGE)
    o.c = __dsub_rn(__dadd_rn(r.obs, r.base_k), r.base_ref);
  else if (KIND == PF_OBS_CARRIER_AFV)
    o.c = __dsub_rn(r.obs, __dmul_rn(fc->clk_anchor[0], o.inv_wl));
  else
    o.c = __dadd_rn(r.obs, __dmul_rn(__dsub_rn(r.base_k, r.base_ref), o.inv_wl));
  o.same = dd && prev && prev->sat_ref[0] == r.sat_ref[0] && prev->sat_ref[1] == r.sat_ref[1] &&
                   prev->sat_ref[2] == r.sat_ref[2]
               ? 1.0
               : 0.0;
  return o;
}

// Residual of one row; rr holds the range to the previous row's reference
// satellite (rows of a constellation share it), and this row's on return.
template <int KIND>
__device__ __forceinline__ double obs_residual(const ObsRow& r, double px, double py, double pz, double clk,
                                               double& rr) {
  const double ax = r.sk[0] - px, ay = r.sk[1] - py, az = r.sk[2] - pz;
  const double rk = sqrt(ax * ax + ay * ay + az * az);
  if constexpr (KIND == PF_OBS_CARRIER_AFV) {
    const double v = r.c - (rk + clk) * r.inv_wl;
    return v - rint(v);
  }
  if (r.same == 0.0) {  // uniform
    const double bx = r.sr[0] - px, by = r.sr[1] - py, bz = r.sr[2] - pz;
    rr = sqrt(bx * bx + by * by + bz * bz);
  }
  if constexpr (KIND == PF_OBS_DD_PSEUDORANGE) return r.c - (rk - rr);
  const double v = r.c - (rk - rr) * r.inv_wl;
  return v - rint(v);
}

__device__ __forceinline__ double obs_cost(const ObsBlock& b, double w, double v) {
  if (b.huber_k > 0.0) {
    const double z = fabs(v) * b.inv_sigma, k = b.huber_k;
    return w * (z < k ? 0.5 * z * z : k * z - 0.5 * k * k);
  }
  return 0.5 * w * v * v * b.inv_sigma2;
}

// One particle per thread and one pass over the rows: the sums over all rows
// and over those inside the gate are formed side by side, and the count of the
// latter chooses one (the gate's test needed a pass of its own before, and every
// row its own reference range).  FP64 roots bound it: 200K particles x 14
// gated rows with two references, 36.4 -> 14.8 us.
template <int KIND, int CAP>
__global__ void __launch_bounds__(kThreads) k_obs_term(EngineDev e, int f, ObsBlock b,
                                                       const __grid_constant__ ObsRowsIn<CAP> in) {
  __shared__ ObsRow s_rows[CAP];
  if (__ldcg(e.err)) return;  // an earlier step's error: reported by the call, the weights stay
  const FilterDesc* fd = e.desc + f;
  const FilterCtrl* fc = e.ctrl + f;
  for (int i = threadIdx.x; i < b.n; i += kThreads)
    s_rows[i] = obs_row<KIND>(fd, fc, in.row[i], i > 0 ? in.row + i - 1 : nullptr);
  __syncthreads();
  const ParticleSrc ps = particle_src(e, fd, fc);
  const bool keep = b.accumulate && fc->lw_zero == 0;
  for (int j = blockIdx.x * kThreads + threadIdx.x; j < ps.n; j += gridDim.x * kThreads) {
    const float* sp = particle_at(e, ps, j);
    const double px = __ldcg(sp), py = __ldcg(sp + e.p_total), pz = __ldcg(sp + 2 * e.p_total),
                 clk = __ldcg(sp + 3 * e.p_total);
    double all = 0.0, inside = 0.0, rr = 0.0;
    int kept = 0;
#pragma unroll 2
    for (int i = 0; i < b.n; ++i) {
      const double v = obs_residual<KIND>(s_rows[i], px, py, pz, clk, rr);
      const double c = obs_cost(b, s_rows[i].w, v);
      all -= c;
      if (!(fabs(v) > b.gate)) inside -= c;
      kept += fabs(v) <= b.gate;
    }
    const double acc = b.gate > 0.0 && kept >= b.gate_min ? inside : all;
    const float l0 = keep ? e.lw[ps.base + j] : 0.f;
    e.lw[ps.base + j] = (float)((double)l0 + acc);
  }
}

}  // namespace pfb
