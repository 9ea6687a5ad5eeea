// pf_velocity.cuh -- per-particle velocity states of the device filter
// (the reference's RBPF-style states, pf_device.cu:67-187 and 610-887):
// a velocity (ECEF, m/s) and its 3x3 covariance per particle, in FP64, held
// in caller-owned device memory beside the engine's particles.
//
// Buffer layout (pf_vel_state_t): two buffers of kVelComp x n doubles,
// component c of particle j at buf[c * n + j]: c = 0..2 velocity, 3..11
// the covariance row-major.  Kernels work on buffer `sel`; the resample
// gather writes the other one.
//
// All arithmetic is FP64 as in the reference.  Particle positions are the
// engine's FP32 offsets about its FP64 anchor (exact in FP64), current
// (gathered through the last resample, if pending).
#pragma once
#include "pf_engine_kernels.cuh"

namespace pfb {

constexpr int kVelComp = 12;
constexpr int kMaxDopplerRows = 64;
constexpr uint32_t TAG_VEL_INIT = 0x06000000u;
constexpr uint32_t TAG_VEL_PREDICT = 0x07000000u;

struct DopplerRow {
  double sat[3];
  double sat_vel[3];
  double doppler_hz;
  double weight;
};

struct DopplerRowsIn {  // a call's rows, as a kernel parameter
  DopplerRow row[kMaxDopplerRows];
};

// Two standard normals from two 32-bit words (Box-Muller in FP64).
__device__ __forceinline__ void normals2_f64(uint32_t a, uint32_t b, double& z0, double& z1) {
  const double two_m32 = 2.3283064365386963e-10;
  const double u1 = ((double)a + 0.5) * two_m32;
  const double u2 = (double)b * two_m32 - 0.5;
  const double r = sqrt(-2.0 * log(u1));
  double s, c;
  sincospi(2.0 * u2, &s, &c);
  z0 = r * c;
  z1 = r * s;
}

// Eight normals for particle slot j from two Philox blocks.
__device__ __forceinline__ void vel_normals(uint32_t j, uint32_t step, uint32_t tag, const FilterDesc* fd,
                                            double (&z)[8]) {
  const U4 r0 = philox10(U4{j, step, tag, (uint32_t)fd->filter_id}, fd->key0, fd->key1);
  const U4 r1 = philox10(U4{j, step, tag | 1u, (uint32_t)fd->filter_id}, fd->key0, fd->key1);
  normals2_f64(r0.x, r0.y, z[0], z[1]);
  normals2_f64(r0.z, r0.w, z[2], z[3]);
  normals2_f64(r1.x, r1.y, z[4], z[5]);
  normals2_f64(r1.z, r1.w, z[6], z[7]);
}

// Velocity v0 (+ spread_vel noise when > 0), covariance init_var * I.
__global__ void __launch_bounds__(kThreads) k_vel_init(EngineDev e, int f, double* vb, double vx, double vy, double vz,
                                                       double spread_vel, double init_var, uint32_t step) {
  const FilterDesc* fd = e.desc + f;
  const int n = fd->n;
  for (int j = blockIdx.x * kThreads + threadIdx.x; j < n; j += gridDim.x * kThreads) {
    double v[3] = {vx, vy, vz};
    if (spread_vel > 0.0) {
      double z[8];
      vel_normals((uint32_t)j, step, TAG_VEL_INIT, fd, z);
      for (int i = 0; i < 3; ++i) v[i] += z[i] * spread_vel;
    }
    for (int i = 0; i < 3; ++i) vb[(size_t)i * n + j] = v[i];
    for (int c = 0; c < 9; ++c) vb[(size_t)(3 + c) * n + j] = (c == 0 || c == 4 || c == 8) ? init_var : 0.0;
  }
}

// Resample gather: out[:, j] = in[:, anc[j]].
__global__ void __launch_bounds__(kThreads) k_vel_gather(EngineDev e, int f, const double* vin, double* vout) {
  const FilterDesc* fd = e.desc + f;
  const int n = fd->n;
  const long long base = fd->p_off;
  const int* seg = seg_markers(e, fd);
  for (int j = blockIdx.x * kThreads + threadIdx.x; j < n; j += gridDim.x * kThreads) {
    int a = ancestor_at(e, seg, base, j);
    a = a < 0 ? 0 : (a >= n ? n - 1 : a);
    for (int c = 0; c < kVelComp; ++c) vout[(size_t)c * n + j] = vin[(size_t)c * n + a];
  }
}

struct VelPredict {
  double guide[3];
  double rot[9];  // ECEF -> local rows (E, N, U)
  double dt, sigma_pos, sigma_vel, alpha, q;
  int kf;
  uint32_t step;
};

// Velocity predict (pf_device.cu:106-187): v = (1 - a) v + a g (+ sigma_vel
// noise unless KF); positions move by v dt + noise, the noise N(0,
// sigma_pos^2 I + dt^2 P_v) (Cholesky) in KF mode, else N(0, sigma_pos^2 I);
// KF mode adds q * dt to the velocity variances.  The positions are read
// through the pending resample gather and written to the other state
// buffer (k_flip_state follows); clocks are copied.
//
// The velocity states follow a pending resample in the same pass (vin != vout:
// read at the ancestor, written in place), so they cross HBM once instead of
// twice, and only the normals in use are drawn.  One particle per thread.  1M
// particles with sampled velocities, gather and predict: 66 -> 43 us; 300K with
// the Kalman covariance 28 -> 14 us.
template <int D, bool KF>
__global__ void __launch_bounds__(kThreads) k_vel_predict(EngineDev e, int f, const double* vin, double* vout,
                                                         VelPredict vp) {
  const FilterDesc* fd = e.desc + f;
  const FilterCtrl* fc = e.ctrl + f;
  const ParticleSrc ps = particle_src(e, fd, fc);
  const int n = ps.n;
  float* dst = (fc->parity ? e.state0 : e.state1) + ps.base;
  const double alpha = fmin(1.0, fmax(0.0, vp.alpha));
  const bool noisy = !KF && vp.sigma_vel > 0.0, moved = vin != vout;
  for (int j = blockIdx.x * kThreads + threadIdx.x; j < n; j += gridDim.x * kThreads) {
    const float* sp = particle_at(e, ps, j);
    const int a = moved ? (int)(sp - (ps.src + ps.base)) : j;
    float x[D];
#pragma unroll
    for (int d = 0; d < D; ++d) x[d] = __ldcg(sp + (size_t)d * e.p_total);
    double v[3], P[9];
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = vin[(size_t)i * n + a];
    if (KF || moved)
#pragma unroll
      for (int c = 0; c < 9; ++c) P[c] = vin[(size_t)(3 + c) * n + a];
    double z[6];
    const U4 r0 = philox10(U4{(uint32_t)j, vp.step, TAG_VEL_PREDICT, (uint32_t)fd->filter_id}, fd->key0, fd->key1);
    normals2_f64(r0.x, r0.y, z[0], z[1]);
    normals2_f64(r0.z, r0.w, z[2], z[3]);
    if (noisy) {
      const U4 r1 = philox10(U4{(uint32_t)j, vp.step, TAG_VEL_PREDICT | 1u, (uint32_t)fd->filter_id}, fd->key0, fd->key1);
      normals2_f64(r1.x, r1.y, z[4], z[5]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      v[i] = (1.0 - alpha) * v[i] + alpha * vp.guide[i];
      if (noisy) v[i] += z[i] * vp.sigma_vel;
      vout[(size_t)i * n + j] = v[i];
    }
    double nz[3];
    if constexpr (KF) {
      const double dt2 = vp.dt * vp.dt, s2 = vp.sigma_pos * vp.sigma_pos;
      const double a00 = s2 + dt2 * P[0], a01 = dt2 * P[1], a02 = dt2 * P[2];
      const double a11 = s2 + dt2 * P[4], a12 = dt2 * P[5], a22 = s2 + dt2 * P[8];
      const double l00 = sqrt(fmax(a00, 0.0));
      double l10 = 0.0, l20 = 0.0;
      if (l00 > 1e-12) {
        l10 = a01 / l00;
        l20 = a02 / l00;
      }
      const double l11 = sqrt(fmax(a11 - l10 * l10, 0.0));
      double l21 = 0.0;
      if (l11 > 1e-12) l21 = (a12 - l20 * l10) / l11;
      const double l22 = sqrt(fmax(a22 - l20 * l20 - l21 * l21, 0.0));
      nz[0] = l00 * z[0];
      nz[1] = l10 * z[0] + l11 * z[1];
      nz[2] = l20 * z[0] + l21 * z[1] + l22 * z[2];
      const double qdt = fmax(vp.q, 0.0) * fmax(vp.dt, 0.0);
      P[0] += qdt;
      P[4] += qdt;
      P[8] += qdt;
    } else {
#pragma unroll
      for (int i = 0; i < 3; ++i) nz[i] = (noisy ? z[3 + i] : z[i]) * vp.sigma_pos;
    }
    if (moved) {
#pragma unroll
      for (int c = 0; c < 9; ++c) vout[(size_t)(3 + c) * n + j] = P[c];
    } else if constexpr (KF) {
      vout[(size_t)3 * n + j] = P[0];
      vout[(size_t)7 * n + j] = P[4];
      vout[(size_t)11 * n + j] = P[8];
    }
    double d[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) d[i] = v[i] * vp.dt + nz[i];
#pragma unroll
    for (int r = 0; r < 3; ++r)
      x[r] = (float)((double)x[r] + vp.rot[3 * r] * d[0] + vp.rot[3 * r + 1] * d[1] + vp.rot[3 * r + 2] * d[2]);
#pragma unroll
    for (int d2 = 0; d2 < D; ++d2) dst[(size_t)d2 * e.p_total + j] = x[d2];
    if (j == n - 1)  // fill the last group of four (EngineDev::state0)
      for (int q = n; q & 3; ++q)
        for (int d2 = 0; d2 < D; ++d2) dst[(size_t)d2 * e.p_total + q] = x[d2];
  }
}

// The particles now sit, gathered, in the other state buffer; the error word goes
// to its pinned mirror.
__global__ void k_flip_state(FilterCtrl* fc, const unsigned* err, unsigned* err_map) {
  fc->parity ^= 1;
  fc->resample_flag = 0;
  *err_map = *err;
}

// ECEF position of local offsets (x, y, z) about the filter's anchor.
__device__ __forceinline__ void particle_ecef(const FilterDesc* fd, const FilterCtrl* fc, float x, float y, float z,
                                              double (&p)[3]) {
  local_to_ecef(fd->rot, fc->anchor, (double)x, (double)y, (double)z, p);
}

struct DopplerArgs {
  int n_sat;
  double wavelength, sigma, gain, max_update;
};

// One row as the kernel uses it: satellite, its velocity, the measured range
// rate -doppler * wavelength, the weight max(w, 0) and (Kalman) sigma^2 / w.
struct DopplerSmem {
  double sat[3], vel[3], rate, w, var;
};

// Unit line of sight from pos to row r's satellite and the rate with the
// satellite's part taken out; false within 1 m (the row is skipped).
__device__ __forceinline__ bool doppler_row(const DopplerSmem& r, const double (&pos)[3], double (&l)[3], double& y) {
  const double dx = r.sat[0] - pos[0], dy = r.sat[1] - pos[1], dz = r.sat[2] - pos[2];
  const double r2 = dx * dx + dy * dy + dz * dz, il = rsqrt(r2);
  l[0] = dx * il;
  l[1] = dy * il;
  l[2] = dz * il;
  y = r.rate - (r.vel[0] * l[0] + r.vel[1] * l[1] + r.vel[2] * l[2]);
  return !(r2 < 1.0);
}

// Doppler terms: pf_device.cu:610-748 (KF false: likelihood with the
// particle's clock drift, then a blend toward its WLS velocity) and
// pf_device.cu:750-887 (KF true: sequential velocity KF, innovation
// likelihood).  Log-weights accumulate (read as zero when reset).
//
// FP64 throughout, and bound by it, so the work is cut to what the result
// needs.  One particle per thread; one reciprocal root per line of sight instead
// of a root and three divisions.
//  * WLS: one pass over the rows instead of three.  With z = y + l.v the row's
//    implied clock drift at the particle's velocity, less that of the first
//    row (so that nothing large is squared), the sums of w, w z, w z^2 give drift
//    and likelihood, and the normal equations of z against (-l, 1) give the
//    velocity correction itself.  The host puts a row of the largest weight
//    first: with z = 0 there, (sum w z)^2 / sum w is at most (1 - w0 / sum w)
//    sum w z^2 (Cauchy and Schwarz), so the difference of the two keeps all but
//    a factor of n rows, whatever the other rows hold (with a first row of weight
//    0 and a Doppler of 1e6 Hz taken instead, log-weights were 8e-4 off).  The
//    equations are solved by LDL^T (the matrix is positive definite: 1e-9 is
//    added to its diagonal, as in the reference, whose unknown is the velocity,
//    hence the right-hand side's 1e-9 terms).
//  * KF: one reciprocal per row; the covariance is symmetric after the first
//    update, so six elements are carried; sum log S as the logarithm of the
//    product of the mantissas plus the exponents.  A row that does not count
//    is selected away instead of branched over, so that the next row's line of
//    sight runs under the serial chain of this one (43 -> 38 us for 300K x 11;
//    lines of sight kept in shared memory from the first pass: 51).
// The chains are long, so warps matter more than registers: 6 CTAs per SM for KF
// (5: 37.4 us, 4: 46, 6 with a few spilled words 36.1), 7 for WLS (the
// compiler's choice: 80.6 us for 1M x 16, 6: 76.0, 7: 74.8, 8: 76.4).
// Kernel time, 1M particles x 16 rows, WLS: 370 -> 72 us; 300K x 11, KF: 92 -> 36.
template <bool KF>
__global__ void __launch_bounds__(128, KF ? 6 : 7) k_doppler(EngineDev e, int f, double* vb,
                                                const __grid_constant__ DopplerRowsIn in, DopplerArgs a) {
  __shared__ DopplerSmem s_rows[kMaxDopplerRows];
  for (int i = threadIdx.x; i < a.n_sat; i += blockDim.x) {
    const DopplerRow& r = in.row[i];
    DopplerSmem& o = s_rows[i];
    for (int k = 0; k < 3; ++k) {
      o.sat[k] = r.sat[k];
      o.vel[k] = r.sat_vel[k];
    }
    o.rate = -r.doppler_hz * a.wavelength;
    o.w = fmax(r.weight, 0.0);
    o.var = o.w > 0.0 ? a.sigma * a.sigma / o.w : 0.0;
  }
  __syncthreads();
  const FilterDesc* fd = e.desc + f;
  const FilterCtrl* fc = e.ctrl + f;
  const int n = fd->n;
  const long long base = fd->p_off;
  const ParticleSrc ps = particle_src(e, fd, fc);
  const bool keep = fc->lw_zero == 0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const float* sp = particle_at(e, ps, j);
    double pos[3];
    particle_ecef(fd, fc, __ldcg(sp), __ldcg(sp + e.p_total), __ldcg(sp + 2 * e.p_total), pos);
    double v[3] = {vb[j], vb[(size_t)n + j], vb[(size_t)2 * n + j]};
    double log_w = 0.0;
    if constexpr (!KF) {
      double sw = 0.0, sz = 0.0, szz = 0.0, z0 = 0.0;
      double sl[3] = {0.0, 0.0, 0.0}, slz[3] = {0.0, 0.0, 0.0};
      double sll[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // xx xy xz yy yz zz
      bool first = true;
      for (int s = 0; s < a.n_sat; ++s) {
        const DopplerSmem& r = s_rows[s];
        double l[3], y;
        if (!doppler_row(r, pos, l, y)) continue;
        double z = y + (l[0] * v[0] + l[1] * v[1] + l[2] * v[2]);
        if (first) z0 = z;
        first = false;
        z -= z0;
        const double w = r.w, wx = w * l[0], wy = w * l[1], wz = w * l[2], wq = w * z;
        sw += w;
        sz += wq;
        szz += wq * z;
        sl[0] += wx;
        sl[1] += wy;
        sl[2] += wz;
        slz[0] += wx * z;
        slz[1] += wy * z;
        slz[2] += wz * z;
        sll[0] += wx * l[0];
        sll[1] += wx * l[1];
        sll[2] += wx * l[2];
        sll[3] += wy * l[1];
        sll[4] += wy * l[2];
        sll[5] += wz * l[2];
      }
      if (sw > 0.0) {
        const double cd = sz / sw;  // drift less z0
        log_w = -0.5 * (szz - cd * sz) / (a.sigma * a.sigma);
        const double gain = fmin(1.0, fmax(0.0, a.gain));
        if (gain > 0.0 && a.n_sat >= 4) {
          // (sum w h h^T + 1e-9 I) (v + dv, z0 + c) = sum w h (z + z0 - l.v), h = (-l, 1)
          const double eps = 1e-9;
          const double a00 = sll[0] + eps, a10 = sll[1], a20 = sll[2], a11 = sll[3] + eps, a21 = sll[4],
                       a22 = sll[5] + eps, a30 = -sl[0], a31 = -sl[1], a32 = -sl[2], a33 = sw + eps;
          const double b0 = -slz[0] - eps * v[0], b1 = -slz[1] - eps * v[1], b2 = -slz[2] - eps * v[2],
                       b3 = sz - eps * z0;
          const double i0 = 1.0 / a00;
          const double l10 = a10 * i0, l20 = a20 * i0, l30 = a30 * i0;
          const double d1 = a11 - l10 * a10, i1 = 1.0 / d1;
          const double m21 = a21 - l20 * a10, m31 = a31 - l30 * a10, l21 = m21 * i1, l31 = m31 * i1;
          const double d2 = a22 - l20 * a20 - l21 * m21, i2 = 1.0 / d2;
          const double m32 = a32 - l30 * a20 - l31 * m21, l32 = m32 * i2;
          const double d3 = a33 - l30 * a30 - l31 * m31 - l32 * m32;
          if (!(a00 < 1e-12) && !(d1 < 1e-12) && !(d2 < 1e-12) && !(d3 < 1e-12)) {
            const double y1 = b1 - l10 * b0, y2 = b2 - l20 * b0 - l21 * y1, y3 = b3 - l30 * b0 - l31 * y1 - l32 * y2;
            const double x3 = y3 / d3, x2 = y2 * i2 - l32 * x3;
            const double x1 = y1 * i1 - l21 * x2 - l31 * x3, x0 = b0 * i0 - l10 * x1 - l20 * x2 - l30 * x3;
            double dv[3] = {x0, x1, x2};
            const double nrm = sqrt(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]);
            if (a.max_update > 0.0 && nrm > a.max_update) {
              const double sc = a.max_update / fmax(nrm, 1e-9);
              for (int i = 0; i < 3; ++i) dv[i] *= sc;
            }
            for (int i = 0; i < 3; ++i) vb[(size_t)i * n + j] = v[i] + gain * dv[i];
          }
        }
      }
    } else {
      double hm[3] = {0.0, 0.0, 0.0}, ym = 0.0, wsum = 0.0;
      for (int s = 0; s < a.n_sat; ++s) {
        const DopplerSmem& r = s_rows[s];
        double l[3], y;
        if (!(r.w > 0.0) || !doppler_row(r, pos, l, y)) continue;
        for (int i = 0; i < 3; ++i) hm[i] -= r.w * l[i];
        ym += r.w * y;
        wsum += r.w;
      }
      if (wsum > 0.0) {
        const double iw = 1.0 / wsum;
        for (int i = 0; i < 3; ++i) hm[i] *= iw;
        ym *= iw;
        double P[9];
        for (int c = 0; c < 9; ++c) P[c] = vb[(size_t)(3 + c) * n + j];
        double pxx = P[0], pxy = P[1], pxz = P[2], pyy = P[4], pyz = P[5], pzz = P[8];
        const bool sym = P[1] == P[3] && P[2] == P[6] && P[5] == P[7];
        double quad = 0.0, mant = 1.0;
        int expo = 0;
        bool any = false;
        auto row = [&](const DopplerSmem& r, auto symc) {
          constexpr bool SYM = decltype(symc)::value;
          double l[3], y;
          const bool use = doppler_row(r, pos, l, y) && r.w > 0.0;
          const double h[3] = {-l[0] - hm[0], -l[1] - hm[1], -l[2] - hm[2]};
          double ph0, ph1, ph2, hp0, hp1, hp2;  // P h and h^T P
          if constexpr (SYM) {
            hp0 = ph0 = pxx * h[0] + pxy * h[1] + pxz * h[2];
            hp1 = ph1 = pxy * h[0] + pyy * h[1] + pyz * h[2];
            hp2 = ph2 = pxz * h[0] + pyz * h[1] + pzz * h[2];
          } else {
            ph0 = P[0] * h[0] + P[1] * h[1] + P[2] * h[2];
            ph1 = P[3] * h[0] + P[4] * h[1] + P[5] * h[2];
            ph2 = P[6] * h[0] + P[7] * h[1] + P[8] * h[2];
            hp0 = h[0] * P[0] + h[1] * P[3] + h[2] * P[6];
            hp1 = h[0] * P[1] + h[1] * P[4] + h[2] * P[7];
            hp2 = h[0] * P[2] + h[1] * P[5] + h[2] * P[8];
          }
          const double S = h[0] * ph0 + h[1] * ph1 + h[2] * ph2 + r.var;
          const bool good = use && S > 1e-18 && isfinite(S);
          const double iS = 1.0 / S;
          const double innov = (y - ym) - (h[0] * v[0] + h[1] * v[1] + h[2] * v[2]);
          const double k0 = ph0 * iS, k1 = ph1 * iS, k2 = ph2 * iS;
          const double v0 = v[0] + k0 * innov, v1 = v[1] + k1 * innov, v2 = v[2] + k2 * innov;
          double nxy, nxz, nyz;
          if constexpr (!SYM) {  // the first update leaves it symmetric
            nxy = 0.5 * ((P[1] - k0 * hp1) + (P[3] - k1 * hp0));
            nxz = 0.5 * ((P[2] - k0 * hp2) + (P[6] - k2 * hp0));
            nyz = 0.5 * ((P[5] - k1 * hp2) + (P[7] - k2 * hp1));
          } else {
            nxy = pxy - k0 * hp1;
            nxz = pxz - k0 * hp2;
            nyz = pyz - k1 * hp2;
          }
          const double nxx = pxx - k0 * hp0, nyy = pyy - k1 * hp1, nzz = pzz - k2 * hp2;
          v[0] = good ? v0 : v[0];
          v[1] = good ? v1 : v[1];
          v[2] = good ? v2 : v[2];
          pxy = good ? (isfinite(nxy) ? nxy : 0.0) : pxy;
          pxz = good ? (isfinite(nxz) ? nxz : 0.0) : pxz;
          pyz = good ? (isfinite(nyz) ? nyz : 0.0) : pyz;
          pxx = good ? ((isfinite(nxx) && nxx > 1e-12) ? nxx : 1e-12) : pxx;
          pyy = good ? ((isfinite(nyy) && nyy > 1e-12) ? nyy : 1e-12) : pyy;
          pzz = good ? ((isfinite(nzz) && nzz > 1e-12) ? nzz : 1e-12) : pzz;
          any |= good;
          quad += good ? innov * innov * iS : 0.0;
          // S is a normal number above 1e-18: mantissa in [1, 2) and exponent
          const long long bits = __double_as_longlong(good ? S : 1.0);
          expo += (int)(bits >> 52) - 1023;
          mant *= __longlong_as_double((bits & 0x000FFFFFFFFFFFFFll) | 0x3FF0000000000000ll);  // <= 2^64
        };
        int s = 0;
        if (!sym)
          while (s < a.n_sat && !any) row(s_rows[s++], std::false_type{});
#pragma unroll 2
        for (; s < a.n_sat; ++s) row(s_rows[s], std::true_type{});
        log_w = -0.5 * (quad + (log(mant) + (double)expo * 0.693147180559945309417));
        for (int i = 0; i < 3; ++i) vb[(size_t)i * n + j] = v[i];
        if (any) {
          const double Q[9] = {pxx, pxy, pxz, pxy, pyy, pyz, pxz, pyz, pzz};
          for (int c = 0; c < 9; ++c) vb[(size_t)(3 + c) * n + j] = Q[c];
        }
      }
    }
    const float l0 = keep ? e.lw[base + j] : 0.f;
    e.lw[base + j] = (float)((double)l0 + log_w);
  }
}

}  // namespace pfb
