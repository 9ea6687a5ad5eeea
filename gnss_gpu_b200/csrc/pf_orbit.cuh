// pf_orbit.cuh -- satellite positions and clocks from broadcast navigation
// records, and the Sagnac-corrected geometric range: the input formation
// upstream of the filter step.
//
//  * Kepler broadcasts (GPS, Galileo, QZSS, BeiDou MEO/IGSO): IS-GPS-200
//    orbit with per-system gravitational parameter, earth rotation rate and
//    relativistic constant (src/ephemeris/ephemeris.cu:14-104 for GPS;
//    python/gnss_gpu/ephemeris.py:36-64,428-512 for the other systems and the
//    BDT offset).
//  * GLONASS: RK4 integration of the PZ-90 equations of motion from the
//    broadcast state, fixed steps plus one residual step
//    (python/gnss_gpu/orbit_glonass.py:67-170).
//  * Sagnac: rotation of the satellite about the earth axis by the signal
//    transit time (python/gnss_gpu/range_model.py:12-40).
//
// FP64 throughout.  The work is O(S) per epoch and small next to the filter step, so
// the kernels batch many epochs into one launch: the broadcast orbits in tiles of
// epochs x satellites (kTileS, kNarrowSats, wide_tiles), the others with a thread per
// (epoch, satellite).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "../../include/gnss_pf_b200.h"

namespace pfb {

constexpr double kWeekSec = 604800.0;
constexpr double kGpstMinusBdt = 14.0;  // gnss_time_scales.py:25
constexpr double kGpstMinusUtc = 18.0;  // gnss_time_scales.py:28
constexpr double kCLight = 299792458.0;
constexpr double kOmegaSagnac = 7.2921151467e-5;  // range_model.py:8

// GLONASS PZ-90 constants (orbit_glonass.py:26-36).
constexpr double kGloRe = 6378136.0;
constexpr double kGloMu = 3.9860044e14;
constexpr double kGloJ2 = 1.0826257e-3;
constexpr double kGloOmega = 7.292115e-5;
constexpr double kGloStep = 60.0;
// Integration steps one record may take: half a week at 1 s per step.
constexpr long kGloMaxSteps = 1L << 20;
// Stored GLONASS states per record and direction (k_glo_table) and the
// scratch they may take per call.
constexpr int kGloTable = 64;
constexpr size_t kGloTableBytes = 64u << 20;

struct OrbitConsts {
  double mu, omega_e, rel_f;
};

// ephemeris.py:55-63: Galileo, QZSS and BeiDou constants; GPS otherwise.
__host__ __device__ inline OrbitConsts orbit_consts(int system) {
  if (system == 'E') return {3.986004418e14, 7.2921151467e-5, -4.442807309e-10};
  if (system == 'C') return {3.986004418e14, 7.292115e-5, -4.442807309e-10};
  return {3.986005e14, 7.2921151467e-5, -4.442807633e-10};  // 'G', 'J' and the rest
}

// gnss_time_scales.py:34-47 (fold into [0, week)).  Finite values only; the
// folding loops are bounded, with fmod past 64 weeks.
__host__ __device__ inline double unwrap_week(double v) {
  if (!isfinite(v)) return v;
  if (fabs(v) > 64.0 * kWeekSec) {
    v = fmod(v, kWeekSec);
    if (v < 0.0) v += kWeekSec;
    return v;
  }
  while (v < 0.0) v += kWeekSec;
  while (v >= kWeekSec) v -= kWeekSec;
  return v;
}

// gnss_time_scales.py:50-63: GPST receive time in the record's time scale.
__host__ __device__ inline double broadcast_rx_sow(int system, double t) {
  if (system == 'C') return unwrap_week(t - kGpstMinusBdt);
  if (system == 'R') return unwrap_week(t - kGpstMinusUtc);
  return t;
}

__host__ __device__ inline double wrap_half_week(double dt) {
  if (dt > kWeekSec / 2.0) dt -= kWeekSec;
  if (dt < -kWeekSec / 2.0) dt += kWeekSec;
  return dt;
}

// (s, c) = (sin x, cos x) -> (sin, cos)(x + d) for |d| <= kSmallAngle: the
// Taylor series of sin d and cos d - 1 (next terms below 1e-24), added to s, c.
constexpr double kSmallAngle = 0.03;
__device__ inline void rotate_small(double& s, double& c, double d) {
  const double d2 = d * d;
  const double sd = d * (1.0 + d2 * (-1.0 / 6.0 + d2 * (1.0 / 120.0 + d2 * (-1.0 / 5040.0 + d2 / 362880.0))));
  const double cd = d2 * (-0.5 + d2 * (1.0 / 24.0 + d2 * (-1.0 / 720.0 + d2 / 40320.0)));
  const double s0 = s;
  s += s0 * cd + c * sd;
  c += c * cd - s0 * sd;
}
// (sin, cos)(x + d) with x's at hand, for any d.
__device__ inline void sincos_near(double sx, double cx, double x, double d, double& s, double& c) {
  if (fabs(d) <= kSmallAngle) {
    s = sx;
    c = cx;
    rotate_small(s, c, d);
  } else {
    sincos(x + d, &s, &c);
  }
}

// 1 / x for x within (1e-30, 1e30): a float reciprocal, refined by Newton's
// method r += r (1 - x r), N times (each doubles its 24 bits).
template <int N>
__device__ inline double recip(double x) {
  double r = (double)__frcp_rn((float)x);
#pragma unroll
  for (int i = 0; i < N; ++i) r = fma(r, fma(-x, r, 1.0), r);
  return r;
}

// sin E and cos E of Kepler's equation by Newton's method from E = M, at
// most 10 updates (ephemeris.cu:14-22, ephemeris.py:417-425).  Sine and cosine
// follow each update by rotation.  Once an update is below 1e-5 the next
// one is below 1e-10: sine and cosine are then evaluated at E, and that last
// update is applied to them (its square is below their rounding).  An update
// needs no more than the leading digits of its divisor.
//
// Where that does not happen (e of about 0.98 and above, no broadcast orbit) the
// updates wander, and the result is E after ten plain ones, stopping below 1e-15:
// whatever E is, a point of the orbit.
__device__ inline void kepler_solve(double M, double e, double& s, double& c) {
  double E = M;
  sincos(M, &s, &c);
  for (int k = 0; k < 10; ++k) {
    const double dE = (M - E + e * s) * recip<0>(1.0 - e * c);
    E += dE;
    if (fabs(dE) < 1e-5) {
      sincos(E, &s, &c);
      const double last = (M - E + e * s) * recip<0>(1.0 - e * c), s0 = s;
      if (!(fabs(last) < 1e-5)) break;
      s += c * last;
      c -= s0 * last;
      return;
    }
    if (fabs(dE) <= kSmallAngle) rotate_small(s, c, dE);
    else sincos(E, &s, &c);
  }
  E = M;
  for (int k = 0; k < 10; ++k) {
    const double dE = (M - E + e * sin(E)) / (1.0 - e * cos(E));
    E += dE;
    if (fabs(dE) < 1e-15) break;
  }
  sincos(E, &s, &c);
}

// What a Kepler record's epochs share.
struct KeplerShared {
  double a, n, sq;        // semi-major axis, mean motion, sqrt(1 - e^2)
  double so, co, si, ci;  // of the argument of perigee and of i0
  double om_rate, om_toe, rel;
};
__device__ inline KeplerShared kepler_shared(const pf_ephemeris_t& k, int system) {
  const OrbitConsts c = orbit_consts(system);
  KeplerShared o;
  o.a = k.sqrt_a * k.sqrt_a;
  o.n = sqrt(c.mu / (o.a * o.a * o.a)) + k.delta_n;
  o.sq = sqrt(1.0 - k.e * k.e);
  sincos(k.omega, &o.so, &o.co);
  sincos(k.i0, &o.si, &o.ci);
  o.om_rate = k.omega_dot - c.omega_e;
  o.om_toe = c.omega_e * k.toe;
  o.rel = c.rel_f * k.e * k.sqrt_a;
  return o;
}

// Position (ECEF, m) and clock correction (s) of a Kepler record at GPST
// second of week t (ephemeris.py:428-512; the GPS-only kernel of
// ephemeris.cu:24-104 is system 'G').  The record's tgd is subtracted as
// stored; callers put the group delay they want there (0 to omit it).
//
// The angles: sine and cosine of the true anomaly are algebraic in those of
// E, the argument of latitude and the inclination are small corrections of
// angles whose sine and cosine are known, so three sincos per epoch (M, E, the
// node) take the place of an arc tangent and some fifteen sines and cosines.
__device__ inline void kepler_orbit(const pf_ephemeris_t& k, const KeplerShared& o, int system, double t, double* pos,
                                    double* clk) {
  const double rx = broadcast_rx_sow(system, t);
  const double tk = wrap_half_week(rx - k.toe);
  double sE, cE;
  kepler_solve(k.M0 + o.n * tk, k.e, sE, cE);
  const double den = 1.0 - k.e * cE, iden = recip<2>(den);
  const double sv = o.sq * sE * iden, cv = (cE - k.e) * iden;
  const double sp = sv * o.co + cv * o.so, cp = cv * o.co - sv * o.so;  // phi = v + omega
  const double s2 = 2.0 * sp * cp, c2 = cp * cp - sp * sp;
  const double du = k.cuc * c2 + k.cus * s2;
  double su = sp, cu = cp;
  if (fabs(du) <= kSmallAngle) rotate_small(su, cu, du);
  else sincos(atan2(sp, cp) + du, &su, &cu);
  const double r = o.a * den + (k.crc * c2 + k.crs * s2);
  double si, ci;
  sincos_near(o.si, o.ci, k.i0, k.idot * tk + (k.cic * c2 + k.cis * s2), si, ci);
  const double xp = r * cu, yp = r * su;
  double sO, cO;
  sincos(k.omega0 + o.om_rate * tk - o.om_toe, &sO, &cO);
  pos[0] = xp * cO - yp * ci * sO;
  pos[1] = xp * sO + yp * ci * cO;
  pos[2] = yp * si;
  const double dt = wrap_half_week(rx - k.toc);
  *clk = k.af0 + k.af1 * dt + k.af2 * dt * dt + o.rel * sE - k.tgd;
}

// PZ-90 equations of motion with the broadcast luni-solar acceleration
// (orbit_glonass.py:67-92): x = (p, v), returns dx/dt.
__device__ inline void glo_deriv(const double* x, const double* acc, double* d) {
  const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
  if (!(r2 > 0.0) || !isfinite(r2)) {
    for (int i = 0; i < 6; ++i) d[i] = 0.0;
    return;
  }
  const double ir = rsqrt(r2), ir2 = ir * ir, ir3 = ir2 * ir;  // one reciprocal root, no division
  const double w2 = kGloOmega * kGloOmega;
  const double at = 1.5 * kGloJ2 * kGloMu * (kGloRe * kGloRe) * ir2 * ir3;
  const double bt = 5.0 * x[2] * x[2] * ir2;
  const double ct = -kGloMu * ir3 - at * (1.0 - bt);
  d[0] = x[3];
  d[1] = x[4];
  d[2] = x[5];
  d[3] = (ct + w2) * x[0] + 2.0 * kGloOmega * x[4] + acc[0];
  d[4] = (ct + w2) * x[1] - 2.0 * kGloOmega * x[3] + acc[1];
  d[5] = (ct - 2.0 * at) * x[2] + acc[2];
}

// One classic RK4 step of h seconds in place (orbit_glonass.py:95-111).
__device__ inline void glo_rk4(double h, double* x, const double* acc) {
  double k1[6], k2[6], k3[6], k4[6], w[6];
  glo_deriv(x, acc, k1);
  for (int i = 0; i < 6; ++i) w[i] = x[i] + k1[i] * (h / 2.0);
  glo_deriv(w, acc, k2);
  for (int i = 0; i < 6; ++i) w[i] = x[i] + k2[i] * (h / 2.0);
  glo_deriv(w, acc, k3);
  for (int i = 0; i < 6; ++i) w[i] = x[i] + k3[i] * h;
  glo_deriv(w, acc, k4);
  for (int i = 0; i < 6; ++i) x[i] += (k1[i] + 2.0 * k2[i] + 2.0 * k3[i] + k4[i]) * (h / 6.0);
}

// Full steps of the GLONASS integration of a record at GPST second of
// week t and what is left for the residual step: what the loop of
// orbit_glonass.py:122-150 leaves, bit for bit.  Returns false past kGloMaxSteps.
//
// With a whole number of seconds per step every difference of the loop is exact (it
// lies on the grid of el's last bit), so the count is a quotient; otherwise the
// loop runs, without its arithmetic (rem decremented in the same order).
__device__ inline bool glo_plan(const pf_glonass_state_t& g, double t, double step, double& el, double& base,
                                long& k, double& rem) {
  el = wrap_half_week(broadcast_rx_sow('R', t) - g.toe);
  base = el < 0.0 ? -step : step;
  rem = el;
  k = 0;
  if (step == rint(step) && fabs(el) < 1e9) {  // |el| <= half a week unless the input is wild
    double q = floor(fabs(el) / step);
    double left = fma(-q, step, fabs(el));
    if (left < 0.0) {  // the quotient was rounded up
      q -= 1.0;
      left += step;
    } else if (left >= step) {
      q += 1.0;
      left -= step;
    }
    if (q > (double)kGloMaxSteps) return false;
    k = (long)q;
    rem = el < 0.0 ? -left : left;
    return true;
  }
  // a NaN time takes no step (the reference returns the broadcast position
  // with a NaN clock); an infinite one runs into the step bound
  while (fabs(rem) >= fabs(base)) {  // |base| >= 1 s, so |rem| > 1e-9 here
    if (++k > kGloMaxSteps) return false;
    rem -= base;
  }
  return true;
}

// GLONASS position and clock at GPST second of week t: align to the
// record's UTC-based scale, integrate from toe in steps of `step` seconds
// with one residual step (orbit_glonass.py:122-170).  `tbl` (may be null)
// holds the states after 1..kc full steps from toe in this direction, shared
// by every epoch of the record: the walk starts from the deepest stored
// state instead of from toe, with the same RK4 steps in the same order, so
// the result is the same bit for bit.  Returns false (outputs NaN) past
// kGloMaxSteps steps.
__device__ inline bool glonass_orbit(const pf_glonass_state_t& g, double t, double step, const double* tbl,
                                     int kc, double* pos, double* clk) {
  double el, base, rem;
  long k;
  if (!glo_plan(g, t, step, el, base, k, rem)) {
    pos[0] = pos[1] = pos[2] = *clk = nan("");
    return false;
  }
  double x[6] = {g.pos[0], g.pos[1], g.pos[2], g.vel[0], g.vel[1], g.vel[2]};
  long done = 0;
  if (tbl && k > 0 && kc > 0) {
    done = k < kc ? k : kc;
    const double* st = tbl + 6 * (done - 1);
    for (int i = 0; i < 6; ++i) x[i] = st[i];
  }
  for (; done < k; ++done) glo_rk4(base, x, g.acc);
  if (fabs(rem) > 1.0e-9) glo_rk4(rem, x, g.acc);
  pos[0] = x[0];
  pos[1] = x[1];
  pos[2] = x[2];
  *clk = -g.tau_n + g.gamma_n * el;
  return true;
}

// Record index of output i (idx null: record s); -1 when out of range.
__device__ inline int orbit_record(const int* idx, long i, int s, int n_recs) {
  const int r = idx ? idx[i] : s;
  return (r < 0 || r >= n_recs) ? -1 : r;
}

// Tiles of 32 EPT epochs x 8 satellites per CTA: a warp takes epochs of one
// satellite, so its lanes run the same orbit model with similar step counts, and
// the CTA's eight satellites make the row-major arrays' segments (8 indexes, 8
// positions, 8 clocks of an epoch) whole sectors.
constexpr int kTileS = 8;
constexpr int kTileThreads = 32 * kTileS;
// Up to this many satellites a tile is 256 EPT epochs x 1 satellite: the warps of
// the missing satellites would only wait.  Whole calls, us, tiles of eight / of one
// (and one thread per satellite-epoch, before the tiles): Kepler 1 x 1M epochs 194 /
// 55 (71), 2 x 500K 112 / 56 (69), 4 x 86,400 40 / 26 (37), GLONASS 1 x 1M 221 / 120
// (201), 4 x 86,400 207 / 114 (308); 1 to 4 x 100 to 3,000 equal.  From five on the
// tiles of eight are ahead of the thread per satellite-epoch (5 x 86,400 42 (43), 7 x
// 86,400 46 (53)) and of the other tile where GLONASS rows are short (7 x 20,000 109
// / 141).
constexpr int kNarrowSats = 4;
// Few epochs of very many satellites leave most lanes of those tiles without an epoch:
// there a tile is one epoch of 256 satellites, a lane per satellite, and so is a warp
// of k_glo_need.  Whole calls, us, tiles of eight / of 256 (and one thread per
// satellite-epoch, before the tiles): Kepler 1 epoch x 8,192 26 / 22 (25), 1 x 100,000
// 194 / 24 (26), 8 x 16,384 37 / 22 (30), 28 x 28,672 71 / 61 (77), 28 x 100,000 219 /
// 182 (218); GLONASS 1 x 100,000 536 / 87 (98), 16 x 50,000 172 / 123 (287).  With fewer
// satellites per epoch the tiles of eight are level or ahead, as GLONASS and Kepler
// records side by side keep a warp of 256's on both paths: 5 x GPS to 3 x GLONASS, 16 x
// 8,192 38 / 47, 16 x 16,384 47 / 49, 16 x 28,672 90 / 72.
inline bool wide_tiles(int n_epoch, int n_sat) {
  return n_epoch <= 28 && n_sat >= 8192 && n_sat >= 1024ll * n_epoch;
}

// Programmatic dependent launch: the state table is needed by GLONASS tiles
// only, so the orbit kernel starts while the table is made.  What the previous
// kernel writes (kmax, tbl) is not read through __restrict__ pointers: such a load
// may take the read-only path, whose lines are not kept in step with other SMs'
// stores, or move above the wait.
__device__ inline void orbit_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ inline void orbit_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Deepest stored state each (GLONASS record, direction) needs: kmax[2r + d]
// >= max over its satellite-epochs of min(full steps, kc).  Whole steps of the
// walk (glo_plan) are at most |el| / step rounded up.  A lane follows its
// satellite through kNeedE / 32 epochs and raises the count of a record when it
// leaves it (an atomic per satellite-epoch took 150 us on a day of 24 satellites).
constexpr int kNeedE = 512;
template <bool WIDE>
__global__ void __launch_bounds__(kTileThreads) k_glo_need(const pf_broadcast_t* __restrict__ recs, int n_recs,
                           const int* __restrict__ idx, const double* __restrict__ times, int n_epoch, int n_sat,
                           double step, int kc, int* __restrict__ kmax) {
  orbit_pdl_trigger();
  const int lane = threadIdx.x & 31, st = (n_sat + kTileS - 1) / kTileS;
  const int s = WIDE ? (int)blockIdx.x * kTileThreads + threadIdx.x
                     : (int)(blockIdx.x % st) * kTileS + (threadIdx.x >> 5);
  const int e0 = WIDE ? 0 : (int)(blockIdx.x / st) * kNeedE;
  const int e1 = s >= n_sat ? e0 : WIDE ? n_epoch : min(n_epoch, e0 + kNeedE);
  int slot = -1, need = 0;
  auto raise = [&](int sl, int m) {
    if (*(volatile int*)(kmax + sl) < m) atomicMax(kmax + sl, m);
  };
  for (int e = WIDE ? e0 : e0 + lane; e < e1; e += WIDE ? 1 : 32) {
    const int r = orbit_record(idx, (long)e * n_sat + s, s, n_recs);
    if (r < 0 || recs[r].system != 'R') continue;
    const double el = wrap_half_week(broadcast_rx_sow('R', times[e]) - recs[r].u.glonass.toe);
    const double k = ceil(fabs(el) / step);
    if (!(k >= 1.0)) continue;  // also NaN
    const int sl = 2 * r + (el < 0.0 ? 1 : 0);
    if (sl != slot) {
      if (slot >= 0) raise(slot, need);
      slot = sl;
      need = 0;
    }
    need = max(need, k < (double)kc ? (int)k : kc);
  }
  __syncwarp();
  const unsigned grp = __match_any_sync(0xffffffffu, slot);
  const int m = (int)__reduce_max_sync(grp, (unsigned)need);
  if (slot >= 0 && lane == __ffs(grp) - 1) raise(slot, m);
}

// The stored states: one thread per (record, direction) integrates kmax
// full steps from toe and keeps every state (6 doubles each, kc per slot).
__global__ void k_glo_table(const pf_broadcast_t* __restrict__ recs, int n_recs, double step,
                            const int* kmax, int kc, double* __restrict__ tbl) {
  orbit_pdl_trigger();
  orbit_pdl_wait();  // kmax
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2 * n_recs) return;
  const int K = __ldcg(kmax + t);
  if (K <= 0 || recs[t >> 1].system != 'R') return;
  const pf_glonass_state_t& g = recs[t >> 1].u.glonass;
  const double h = (t & 1) ? -step : step;
  double x[6] = {g.pos[0], g.pos[1], g.pos[2], g.vel[0], g.vel[1], g.vel[2]};
  double* out = tbl + (size_t)t * kc * 6;
  for (int k = 0; k < K; ++k) {
    glo_rk4(h, x, g.acc);
    for (int c = 0; c < 6; ++c) out[6 * k + c] = x[c];
  }
}

// Multi-system records: out[e][s] from recs[idx[e*S+s]] (or recs[s] when idx
// is null) at times[e]; an index outside [0, n_recs) gives NaN, and so does a
// GLONASS integration past kGloMaxSteps steps (also flagged in *err if given).
// tbl / kc: the GLONASS state table of k_glo_table, or null / 0.
//
// FP64 bound (36 bytes a satellite-epoch are 31 us of the day-long call at
// the measured copy rate).  Each thread takes EPT epochs of its satellite and
// keeps what its record's epochs share; results go through shared memory, so
// that positions and clocks leave as whole rows of TS satellites.  A day at
// 1 Hz of 40 Kepler and 24 GLONASS satellites, the whole call: 495 -> 247 us.
// Four CTAs per SM (64 registers): with two 291 us, with three 258.
template <int EPT, int TS>
__global__ void __launch_bounds__(kTileThreads, 4) k_broadcast_orbits(const pf_broadcast_t* __restrict__ recs, int n_recs,
                                   const int* __restrict__ idx, const double* __restrict__ times,
                                   int n_epoch, int n_sat, double glo_step, const double* tbl, int kc,
                                   double* __restrict__ pos, double* __restrict__ clk, int* __restrict__ err) {
  constexpr bool kWide = TS == kTileThreads;  // lanes along the satellites of one epoch
  constexpr int kRows = kTileThreads / TS, kE = kRows * EPT;  // epochs at a time, and of the tile
  __shared__ int s_idx[kE][TS + 1];
  __shared__ double s_pos[kRows][3 * TS + 1];
  __shared__ double s_clk[kRows][TS + 1];
  const int w = kWide ? threadIdx.x : (threadIdx.x >> 5) % TS;
  const int row = kWide ? 0 : (threadIdx.x >> 5) / TS * 32 + (threadIdx.x & 31);
  const int st = (n_sat + TS - 1) / TS, et = (n_epoch + kE - 1) / kE;
  // satellites slowest: GLONASS satellites, mostly at the end of the list,
  // come last and find their table ready
  const int s0 = (int)(blockIdx.x / et) * TS, e0 = (int)(blockIdx.x % et) * kE;
  const int ns = min(TS, n_sat - s0);
  if (s0 >= st * TS) return;
  for (int i = threadIdx.x; i < kE * TS; i += kTileThreads) {
    const int e = e0 + i / TS, s = s0 + i % TS;
    s_idx[i / TS][i % TS] = e < n_epoch && s < n_sat ? orbit_record(idx, (long)e * n_sat + s, s, n_recs) : -1;
  }
  __syncthreads();
  KeplerShared sh;
  int have = -1;
  bool waited = false;
#pragma unroll 1
  for (int q = 0; q < EPT && e0 + kRows * q < n_epoch; ++q) {
    const int e = e0 + kRows * q + row, r = s_idx[kRows * q + row][w];
    double p[3], c;
    p[0] = p[1] = p[2] = c = nan("");
    const bool glo = r >= 0 && recs[r].system == 'R';
    if (tbl && !waited && __any_sync(0xffffffffu, glo)) {
      orbit_pdl_wait();
      waited = true;
    }
    if (glo) {
      const pf_glonass_state_t& g = recs[r].u.glonass;
      const double el = wrap_half_week(broadcast_rx_sow('R', times[e]) - g.toe);
      const double* tb = tbl ? tbl + ((size_t)2 * r + (el < 0.0 ? 1 : 0)) * kc * 6 : nullptr;
      if (!glonass_orbit(g, times[e], glo_step, tb, kc, p, &c) && err) atomicOr(err, 1);
    } else if (r >= 0) {
      const pf_ephemeris_t& k = recs[r].u.kepler;
      if (r != have) {
        sh = kepler_shared(k, recs[r].system);
        have = r;
      }
      kepler_orbit(k, sh, recs[r].system, times[e], p, &c);
    }
    __syncthreads();  // the previous rows have left
    s_pos[row][3 * w] = p[0];
    s_pos[row][3 * w + 1] = p[1];
    s_pos[row][3 * w + 2] = p[2];
    s_clk[row][w] = c;
    __syncthreads();
    const int rows = min(kRows, n_epoch - (e0 + kRows * q));
    const long row0 = (long)(e0 + kRows * q) * n_sat + s0;
    if (pos)
      for (int i = threadIdx.x; i < rows * 3 * TS; i += kTileThreads) {
        const int er = i / (3 * TS), k = i % (3 * TS);
        if (k < 3 * ns) pos[3 * (row0 + (long)er * n_sat) + k] = s_pos[er][k];
      }
    if (clk)
      for (int i = threadIdx.x; i < rows * TS; i += kTileThreads)
        if (i % TS < ns) clk[row0 + (long)(i / TS) * n_sat + i % TS] = s_clk[i / TS][i % TS];
  }
  if (tbl && !waited) orbit_pdl_wait();  // the grid ends after the table's
}

// GPS-constant batch over the reference's parameter array
// (ephemeris.cu:106-180): out[e][s] from params[s] at times[e].
__global__ void k_sat_pos_gps(const pf_ephemeris_t* __restrict__ params, const double* __restrict__ times,
                              int n_epoch, int n_sat, double* __restrict__ pos, double* __restrict__ clk) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)n_epoch * n_sat) return;
  const int e = (int)(i / n_sat), s = (int)(i - (long)e * n_sat);
  double p[3], c;
  kepler_orbit(params[s], kepler_shared(params[s], 'G'), 'G', times[e], p, &c);
  pos[3 * i] = p[0];
  pos[3 * i + 1] = p[1];
  pos[3 * i + 2] = p[2];
  clk[i] = c;
}

// Sagnac rotation and range (range_model.py:12-40) for receivers rx[e] and
// satellites sat[e][s]: theta = omega_e |rx - sat| / c about the z axis.
__global__ void k_sagnac(const double* __restrict__ rx, const double* __restrict__ sat, int n_epoch, int n_sat,
                         double* __restrict__ sat_rot, double* __restrict__ range) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)n_epoch * n_sat) return;
  const long e = i / n_sat;
  const double r0 = rx[3 * e], r1 = rx[3 * e + 1], r2 = rx[3 * e + 2];
  const double s0 = sat[3 * i], s1 = sat[3 * i + 1], s2 = sat[3 * i + 2];
  const double d0 = r0 - s0, d1 = r1 - s1, d2 = r2 - s2;
  const double th = kOmegaSagnac * (sqrt(d0 * d0 + d1 * d1 + d2 * d2) / kCLight);
  const double ct = cos(th), st = sin(th);
  const double x = s0 * ct + s1 * st, y = -s0 * st + s1 * ct;
  if (sat_rot) {
    sat_rot[3 * i] = x;
    sat_rot[3 * i + 1] = y;
    sat_rot[3 * i + 2] = s2;
  }
  if (range) {
    const double q0 = r0 - x, q1 = r1 - y, q2 = r2 - s2;
    range[i] = sqrt(q0 * q0 + q1 * q1 + q2 * q2);
  }
}

// WGS84 geodetic latitude, longitude (rad) and height of ECEF points by
// Bowring's closed form (src/utils/coordinates.cu:7-27): one auxiliary
// angle, no iteration.
constexpr double kWgsA = 6378137.0;
constexpr double kWgsF = 1.0 / 298.257223563;
constexpr double kWgsB = kWgsA * (1.0 - kWgsF);
constexpr double kWgsE2 = 2.0 * kWgsF - kWgsF * kWgsF;

__global__ void k_ecef_to_lla(const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ z, double* __restrict__ lat, double* __restrict__ lon,
                              double* __restrict__ alt, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double X = x[i], Y = y[i], Z = z[i];
  const double p = sqrt(X * X + Y * Y);
  const double th = atan2(Z * kWgsA, p * kWgsB);
  const double st = sin(th), ct = cos(th);
  const double la = atan2(Z + kWgsE2 / (1.0 - kWgsE2) * kWgsB * st * st * st, p - kWgsE2 * kWgsA * ct * ct * ct);
  const double sl = sin(la);
  lat[i] = la;
  lon[i] = atan2(Y, X);
  alt[i] = p / cos(la) - kWgsA / sqrt(1.0 - kWgsE2 * sl * sl);
}

}  // namespace pfb
