// pf_generic.cuh -- the device filter's likelihood family (weight mode
// PF_WEIGHT_GENERIC), selected per call with pfe_set_likelihood:
//
//   Gaussian      -w r^2 / (2 sigma^2)                                     (pf_device.cu:273-275)
//   Student's t   -(nu + 1)/2 log(1 + w r^2 / (nu sigma^2))                (pf_device.cu:265-266)
//   Huber         -w rho_k(|r| / sigma)                                    (pf_device.cu:19-26,267-268)
//   GMM           log(w_los N(r; 0, sigma) + (1 - w_los) N(r; mu, s_nlos)),
//                 each quadratic term scaled by w                           (pf_device.cu:373-436)
//
// with an optional per-particle NLOS gate (pf_device.cu:236-258): a particle
// drops the satellites whose |r| exceeds the gate, unless fewer than
// min(n_sat, 4) would remain, in which case it keeps all of them.
//
// The residual r is the epoch kernel's second-order form (sat_pair_update).
// Satellite table entries use the mixture layout (kMixStride float2):
//   eE eN | eU g/2 | y w | c0 c1 | c2 c3 | mu mode
// GMM: c0 = log w_los - log sigma, c1 = -w / (2 sigma^2), c2, c3 the NLOS pair, -mu
// in the place of mu; Huber: none; Student's t: c1 = w / (nu
// sigma^2); Gaussian: c1 = -w / (2 sigma^2).  One likelihood holds for every
// satellite, and one of weight <= 0 gets constants that add nothing and a finite
// residual (its record may hold anything), so the loops are free of branches.
#pragma once
#include "pf_learned.cuh"

namespace pfb {

// Table entry of one satellite for the generic likelihood.
__device__ __forceinline__ void write_generic_entry(float2* o, const EngineDev& e, float sigma, float eE, float eN,
                                                    float eU, float g, float y, float w) {
  const bool used = w > 0.f;
  o[0] = bc(used ? eE : 0.f); o[1] = bc(used ? eN : 0.f); o[2] = bc(used ? eU : 0.f); o[3] = bc(used ? 0.5f * g : 0.f);
  o[4] = bc(used ? y : 0.f); o[5] = bc(used ? w : 0.f);
  float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f, mu = 0.f;
  const float s2 = sigma * sigma;
  if (e.lk_type == PF_LIK_GMM) {
    const float sn = e.lk_sigma_nlos;
    c2 = -INFINITY;  // unused: log(e^0 + 0)
    if (used) {
      c0 = logf(e.lk_w_los) - logf(sigma);
      c1 = -0.5f * w / s2;
      c2 = logf(1.f - e.lk_w_los) - logf(sn);
      c3 = -0.5f * w / (sn * sn);
      mu = e.lk_mu_nlos;
    }
  } else if (!used) {
  } else if (e.lk_type == PF_LIK_STUDENT_T) {
    c1 = w / (e.lk_nu * s2);
  } else if (e.lk_type == PF_LIK_GAUSSIAN) {
    c1 = -0.5f * w / s2;
  }
  o[6] = bc(c0); o[7] = bc(c1); o[8] = bc(c2); o[9] = bc(c3);
  o[10] = bc(-mu); o[11] = bc(0.f);
}

// Residual of two particles for one table entry (as sat_pair_update).
__device__ __forceinline__ float2 entry_residual(const float2* entry, float2 dx, float2 dy, float2 dz, float2 nbb,
                                                 float2 ncb) {
  const float4* sv = reinterpret_cast<const float4*>(entry);
  const float4 q0 = sv[0], q1 = sv[1], q2 = sv[2];
  const float2 eE = f2(q0.x, q0.y), eN = f2(q0.z, q0.w), eU = f2(q1.x, q1.y), g2 = f2(q1.z, q1.w);
  const float2 yc = __fadd2_rn(f2(q2.x, q2.y), ncb);
  float2 ye = __ffma2_rn(eE, dx, yc);
  ye = __ffma2_rn(eN, dy, ye);
  ye = __ffma2_rn(eU, dz, ye);
  const float2 ed = __ffma2_rn(yc, bc(-1.0f), ye);
  const float2 sq = __ffma2_rn(ed, ed, nbb);
  return __ffma2_rn(sq, g2, ye);
}

template <int T>
struct LikType {
  static constexpr int value = T;
};

// Adds the satellites [s0, s1) of the table to two particle pairs; a residual
// beyond lim[k] (infinite without the gate) is dropped.
template <int TYPE>
__device__ __forceinline__ void generic_pairs(const float2* s_sat, int s0, int s1, const float2 (&dx)[2],
                                              const float2 (&dy)[2], const float2 (&dz)[2], const float2 (&nbb)[2],
                                              const float2 (&ncb)[2], float2 (&lwp)[2], const float (&lim)[4],
                                              float huber_k, float inv_sigma, float t_scale) {
#pragma unroll 2
  for (int s = s0; s < s1; ++s) {
    const float2* entry = s_sat + kMixStride * s;
    const float4* sv = reinterpret_cast<const float4*>(entry);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float2 r = entry_residual(entry, dx[p], dy[p], dz[p], nbb[p], ncb[p]);
      const bool o0 = fabsf(r.x) > lim[2 * p], o1 = fabsf(r.y) > lim[2 * p + 1];
      if constexpr (TYPE == PF_LIK_GAUSSIAN) {
        const float4 q3 = sv[3];
        const float2 rk = f2(o0 ? 0.f : r.x, o1 ? 0.f : r.y);
        lwp[p] = __ffma2_rn(__fmul2_rn(f2(q3.z, q3.w), rk), rk, lwp[p]);
      } else if constexpr (TYPE == PF_LIK_HUBER) {
        const float4 q2 = sv[2];
        huber_pair(f2(o0 ? 0.f : r.x, o1 ? 0.f : r.y), q2.z, huber_k, inv_sigma, lwp[p]);
      } else if constexpr (TYPE == PF_LIK_STUDENT_T) {
        const float4 q3 = sv[3];
        const float2 rk = f2(o0 ? 0.f : r.x, o1 ? 0.f : r.y);
        const float2 q = __ffma2_rn(__fmul2_rn(f2(q3.z, q3.w), rk), rk, bc(1.f));  // >= 1
        lwp[p] = __ffma2_rn(bc(t_scale), __fmul2_rn(f2(lg2_normal(q.x), lg2_normal(q.y)), bc(0.693147180559945309f)),
                            lwp[p]);
      } else {
        const float4 q3 = sv[3], q4 = sv[4], q5 = sv[5];
        const float2 a = __ffma2_rn(__fmul2_rn(f2(q3.z, q3.w), r), r, f2(q3.x, q3.y));
        const float2 dm = __fadd2_rn(r, f2(q5.x, q5.y));
        const float2 b = __ffma2_rn(__fmul2_rn(f2(q4.z, q4.w), dm), dm, f2(q4.x, q4.y));
        const float2 l = log_add_pair(a, b);
        lwp[p] = __fadd2_rn(lwp[p], f2(o0 ? 0.f : l.x, o1 ? 0.f : l.y));
      }
    }
  }
}

// Satellites of [s0, s1) with |r| <= gate, per particle (for the gate).
__device__ __forceinline__ void generic_kept(const float2* s_sat, int s0, int s1, const float2 (&dx)[2],
                                             const float2 (&dy)[2], const float2 (&dz)[2], const float2 (&nbb)[2],
                                             const float2 (&ncb)[2], int (&kept)[4], int& used, float gate) {
  for (int s = s0; s < s1; ++s) {
    const float2* entry = s_sat + kMixStride * s;
    ++used;  // every satellite counts, as in the reference
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const float2 r = entry_residual(entry, dx[p], dy[p], dz[p], nbb[p], ncb[p]);
      kept[2 * p] += fabsf(r.x) <= gate;
      kept[2 * p + 1] += fabsf(r.y) <= gate;
    }
  }
}

}  // namespace pfb
