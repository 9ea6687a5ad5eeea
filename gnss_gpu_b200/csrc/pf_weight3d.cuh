// pf_weight3d.cuh -- the engine's building-aware likelihood and the
// line-of-sight queries over a device mesh (hierarchy and traversal in
// pf_bvh.cuh).
#pragma once
#include "pf_bvh.cuh"
#include "pf_engine_kernels.cuh"

namespace pfb {

// Building-aware pseudorange likelihood (weight_3d.cu:86-177): per
// satellite a ray from the particle; blocked rays use the NLOS-prior
// p_blocked, clear ones p_clear, in a mixture of a tight LOS Gaussian and a
// wide NLOS Gaussian whose positive residuals are reduced by nlos_bias.
//
// Shadow cells.  A million walks of the hierarchy per satellite would ask
// nearly the same question a million times: the cloud is a few metres wide.
// So the cloud's box is cut into cells and these into blocks of 4 x 4 x 2, and
// the rays from a block (a cell) to a satellite are treated as one beam:
//   k_cells_box     mean and spread of the particles' offsets -> the grid, or none
//                   for a cloud too wide for cells (kCellSpan)
//   k_cells_mark    which blocks hold particles
//   k_cells_block   per (block, satellite) one walk of the hierarchy with the
//                   beam's centre ray and boxes enlarged by its half extents;
//                   triangles that no ray can hit are dropped, one that every
//                   ray hits settles the block, the others are listed
//   k_cells_cell    per (cell, satellite) the listed triangles again, with the
//                   cell's thinner beam: blocked, clear, or a mask of the
//                   triangles that some ray may hit
//   k_weight_3d     per particle the verdicts of its cell; where triangles are
//                   left, the particle's own ray is tested against them
//                   (collected per warp, so the tests run on full warps)
// A particle outside the grid, or in a block with a long list, walks the
// hierarchy with its own ray.  The verdict on every ray is that of its own
// ray-triangle tests, whatever the grid.
//
// Why the bounds hold.  With c the centre of the cell, h its half extents
// and L the distance from c to the satellite, |o_i - c| <= h per component
// and |d_i - d_c| <= 2 |h| / L, so at any t <= T ray i is within
//   H = h + 2 T |h| / L (+ rounding)
// of the centre ray at the same t (T: the farthest point of the mesh, or the
// satellite).  Hence a box hit by ray i, enlarged by H, is hit by the centre
// ray; and where ray i meets a triangle's plane, its barycentric coordinates
// and distance are those of a ray from c + eta along d_c with |eta| <= H, which
// are linear in eta.
constexpr int kBeamCap = 30;                  // triangles of a block's list
constexpr unsigned kCodeBlocked = 1u << 31;   // a cell's code: the mask of its triangles in the block's list,
constexpr unsigned kCodePerRay = 1u << 30;    // or one of these
constexpr int kBlockCells = 32;               // 4 x 4 x 2
constexpr int kCellsMax = 1 << 18;            // cells of a grid
constexpr int kCellItems = 1 << 22;           // cells x satellites
constexpr int kBoxSample = 1 << 16;           // particles that place the grid
// Rays (particles x satellites) up to which each gets its own thread, and above
// which the cells pay.  Likelihood alone, us, one thread per particle / this
// rule: 3,000 x 16 95 / 42, 10,000 x 24 132 / 53, 60,000 x 16 132 / 122, 180,000 x
// 16 256 / 137, 500,000 x 16 541 / 213, 1M x 16 963 / 225 to 330 (the wider the
// cloud the more); 200,000 x 10, 125 / 140 with cells, hence the line above it.
constexpr long long kThreadRays = 1000000;
constexpr long long kCellRays = 2200000;
// Cells wider than this share of the spacing of the mesh's triangles settle too
// little: most lists overflow or hold many triangles per ray, and every particle
// walks its own rays instead (n_blocks = 0).  The cloud's width is known on the
// device only, so both kernels are launched and one returns at once.  Likelihood
// alone, us, walks / cells: city of 2,490 triangles at 40 m spacing, 1M x 16
// particles spread by 50, 100, 140, 200, 300 m (cells of 0.18, 0.36, 0.50, 0.72,
// 1.07 spacings) 1213 / 614, 1285 / 923, 1263 / 1103, 1233 / 2333, 1187 / 2975; the
// same triangles in four, 1M, 0.36 and 0.50 spacings 1559 / 1006, 1591 / 1967; 200K x
// 16, 0.28 and 0.55 spacings 328 / 246, 351 / 352.  A cloud sent back costs some 20 us
// over the walks (300 m: 1206 us, 150K x 16 particles 263 against 241).
constexpr float kCellSpan = 0.45f;
#ifndef PF_CELL_PARTICLES
#define PF_CELL_PARTICLES 8
#endif

// Cells to aim at over the whole grid; it may come out a quarter larger.
inline __host__ __device__ int cells_wanted(int n, int n_sat) {
  const int c = n / PF_CELL_PARTICLES * 9 / 4;  // (8.4 / 6.4)^3
  const int most = kCellItems / n_sat < kCellsMax ? kCellItems / n_sat : kCellsMax;
  const int least = c < 32768 ? 32768 : c;  // few particles: the cells stay as thin
  return least < most / 5 * 4 ? least : most / 5 * 4;
}

// The grid of a call, in the filter's local frame.
struct CellGrid {
  float lo[3];
  float side, inv_side;
  int bdim[3];   // blocks
  int n_blocks;  // 0: no cells, the particles walk
  float M[9];    // local offsets -> mesh frame: M x + off
  float off[3];
  float hm[3];   // |M| (1, 1, 1)
  float hb[3];   // |M| (4, 4, 2)
  unsigned ticket;
  unsigned long long count;
  long long s1[3], s2[3];  // sums of the offsets and of their squares, cm
};

// A block's list for one satellite.
struct BlockList {
  unsigned n;  // triangles, or kCodeBlocked, kCodePerRay
  float ext;   // enlargement of the beam beyond the box's half extents
  int tri[kBeamCap];
};

// Scratch of a call.
struct CellBufs {
  CellGrid* grid;
  unsigned* mark;   // a bit per block: holds particles
  unsigned* code;   // [cells][satellites]
  BlockList* list;  // [blocks][satellites]
  unsigned* blk;    // instead of cells: bit j % 32 of word [satellite][j / 32], the ray of particle j is blocked
};
enum RayMode : int { RAYS_WALK = 0, RAYS_CELLS = 1, RAYS_WORDS = 2 };

struct Beam {
  float3 c, d, H;
  float t_lo, t_hi;  // a triangle nearer than t_lo is in front of the satellite for every ray, beyond t_hi for none
};

// 0: no ray of the beam hits the triangle, 1: some may, 2: all do.  (As
// tri_hit, the barycentric coordinates u, v, w = 1 - u - v and the distance t
// of the centre ray, each with its variation over the beam.)
__device__ __forceinline__ int beam_triangle(const Beam& b, const float4 v0, const float4 e1, const float4 e2) {
  const float3 d = b.d, H = b.H;
  const float hx = d.y * e2.z - d.z * e2.y, hy = d.z * e2.x - d.x * e2.z, hz = d.x * e2.y - d.y * e2.x;
  const float a = e1.x * hx + e1.y * hy + e1.z * hz;
  const float n1 = e1.x * e1.x + e1.y * e1.y + e1.z * e1.z, n2 = e2.x * e2.x + e2.y * e2.y + e2.z * e2.z;
  const bool steep = a * a > 1e-4f * n1 * n2;  // else grazing or degenerate: left to the rays
  const float f = 1.0f / a, af = fabsf(f), m = 2e-3f;
  const float sx = b.c.x - v0.x, sy = b.c.y - v0.y, sz = b.c.z - v0.z;
  const float u = f * (sx * hx + sy * hy + sz * hz);
  const float qx = sy * e1.z - sz * e1.y, qy = sz * e1.x - sx * e1.z, qz = sx * e1.y - sy * e1.x;
  const float v = f * (d.x * qx + d.y * qy + d.z * qz), w = 1.0f - u - v;
  const float t = f * (e2.x * qx + e2.y * qy + e2.z * qz);
  const float gx = e1.y * d.z - e1.z * d.y, gy = e1.z * d.x - e1.x * d.z, gz = e1.x * d.y - e1.y * d.x;
  const float nx = e1.y * e2.z - e1.z * e2.y, ny = e1.z * e2.x - e1.x * e2.z, nz = e1.x * e2.y - e1.y * e2.x;
  const float du = af * (fabsf(hx) * H.x + fabsf(hy) * H.y + fabsf(hz) * H.z) + m;
  const float dv = af * (fabsf(gx) * H.x + fabsf(gy) * H.y + fabsf(gz) * H.z) + m;
  const float dw = af * (fabsf(hx + gx) * H.x + fabsf(hy + gy) * H.y + fabsf(hz + gz) * H.z) + m;
  const float dt = af * (fabsf(nx) * H.x + fabsf(ny) * H.y + fabsf(nz) * H.z) + 0.01f;
  const bool miss = u + du < 0.f || u - du > 1.f || v + dv < 0.f || w + dw < 0.f || t + dt < 0.f || t - dt > b.t_hi;
  const bool full = u - du > 0.f && v - dv > 0.f && w - dw > 0.f && t - dt > 0.f && t + dt < b.t_lo;
  return !steep ? 1 : miss ? 0 : full ? 2 : 1;
}

// slab() for the beam: the box enlarged by H, as cp = c + H, cm = c - H.
__device__ __forceinline__ bool beam_slab(const float4 mn, const float4 mx, const float3 cp, const float3 cm,
                                          const float3 inv, float tmax, float& tin) {
  float a = (mn.x - cp.x) * inv.x, b = (mx.x - cm.x) * inv.x;
  float t0 = fmaxf(0.f, fminf(a, b)), t1 = fminf(tmax, fmaxf(a, b));
  a = (mn.y - cp.y) * inv.y;
  b = (mx.y - cm.y) * inv.y;
  t0 = fmaxf(t0, fminf(a, b));
  t1 = fminf(t1, fmaxf(a, b));
  a = (mn.z - cp.z) * inv.z;
  b = (mx.z - cm.z) * inv.z;
  t0 = fmaxf(t0, fminf(a, b));
  t1 = fminf(t1, fmaxf(a, b));
  tin = t0;
  return t0 <= t1;
}

__device__ __forceinline__ float keep_off_zero(float v) { return copysignf(fmaxf(fabsf(v), 1e-9f), v); }

// The beam from the box c +- h, enlarged by ext, to the satellite at `sat`
// (mesh frame), L away.
__device__ __forceinline__ Beam make_beam(const float3 c, const float3 h, const float3 sat, float L, float ext) {
  const float il = 1.0f / L, slack = sqrtf(h.x * h.x + h.y * h.y + h.z * h.z) + 0.01f + 1e-6f * L;
  Beam b;
  b.c = c;
  b.d = make_float3(keep_off_zero((sat.x - c.x) * il), keep_off_zero((sat.y - c.y) * il),
                    keep_off_zero((sat.z - c.z) * il));
  b.H = make_float3(h.x + ext, h.y + ext, h.z + ext);
  b.t_lo = L - slack;
  b.t_hi = L + slack;
  return b;
}
__device__ __forceinline__ float dist3(const float3 a, const float3 b) {
  const float x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
  return sqrtf(x * x + y * y + z * z);
}

// Walks the hierarchy with the beam from the box c +- h to the satellite and
// fills the block's list.
__device__ __forceinline__ void beam_walk(const MeshDev& m, const float3 c, const float3 h, const float3 sat,
                                          BlockList* out) {
  const float L = dist3(sat, c), nh = sqrtf(h.x * h.x + h.y * h.y + h.z * h.z);
  if (!(L > 4.f * nh + 0.1f) || !(L < 1e12f)) {
    out->n = kCodePerRay;
    return;
  }
  // farthest corner of the mesh (an unused child of a single-leaf root is at 1e30)
  float T = 0.f;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float4 mn = __ldg(m.nodes + 2 * k), mx = __ldg(m.nodes + 2 * k + 1);
    if (mn.x < 1e29f) {
      const float fx = fmaxf(fabsf(mn.x - c.x), fabsf(mx.x - c.x)), fy = fmaxf(fabsf(mn.y - c.y), fabsf(mx.y - c.y)),
                  fz = fmaxf(fabsf(mn.z - c.z), fabsf(mx.z - c.z));
      T = fmaxf(T, sqrtf(fx * fx + fy * fy + fz * fz));
    }
  }
  T = fminf(L, T) + nh + 1.f;
  const float ext = T * (2.f * nh / L) + 0.01f + 2e-6f * T;
  const Beam b = make_beam(c, h, sat, L, ext);
  out->ext = ext;
  const float3 inv = make_float3(1.0f / b.d.x, 1.0f / b.d.y, 1.0f / b.d.z);
  const float3 cp = make_float3(c.x + b.H.x, c.y + b.H.y, c.z + b.H.z);
  const float3 cm = make_float3(c.x - b.H.x, c.y - b.H.y, c.z - b.H.z);
  int stack[kBvhStack];
  int sp = 0, node = 0;
  unsigned cnt = 0;
  for (int visits = 0; visits <= m.n_nodes; ++visits) {  // bound as in bvh_blocked
    if ((unsigned)node >= (unsigned)m.n_nodes) break;
    const float4* nd = m.nodes + 4 * node;
    const float4 l0 = __ldg(nd), l1 = __ldg(nd + 1), r0 = __ldg(nd + 2), r1 = __ldg(nd + 3);
    float tl, tr;
    const int cl = __float_as_int(l0.w), cr = __float_as_int(l1.w);
    bool hl = beam_slab(l0, l1, cp, cm, inv, b.t_hi, tl), hr = beam_slab(r0, r1, cp, cm, inv, b.t_hi, tr);
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {  // leaves among the two children
      const int ref = side ? cr : cl;
      if (!(side ? hr : hl) || ref >= 0) continue;
      if (side) hr = false;
      else hl = false;
      const int code = ~ref, s0 = code >> 3, n = (code & 7) + 1;
      if (s0 + n > m.n_tris) continue;  // malformed reference
      // the leaf's triangles side by side: their loads and tests overlap
      float4 t[kBvhLeaf][3];
      int r[kBvhLeaf];
#pragma unroll
      for (int k = 0; k < kBvhLeaf; ++k) {
        const float4* q = m.tris + 3 * (s0 + min(k, n - 1));
        t[k][0] = __ldg(q);
        t[k][1] = __ldg(q + 1);
        t[k][2] = __ldg(q + 2);
      }
      bool all = false;
#pragma unroll
      for (int k = 0; k < kBvhLeaf; ++k) {
        r[k] = beam_triangle(b, t[k][0], t[k][1], t[k][2]);
        all = all || r[k] == 2;
      }
      if (all) {
        out->n = kCodeBlocked;
        return;
      }
#pragma unroll
      for (int k = 0; k < kBvhLeaf; ++k)
        if (r[k] == 1 && k < n) {
          if (cnt == kBeamCap) {
            out->n = kCodePerRay;
            return;
          }
          out->tri[cnt++] = s0 + k;
        }
    }
    if (hl && hr) {
      const bool lf = tl <= tr;
      if (sp < kBvhStack) stack[sp++] = lf ? cr : cl;
      node = lf ? cl : cr;
    } else if (hl) {
      node = cl;
    } else if (hr) {
      node = cr;
    } else {
      if (sp == 0) {
        out->n = cnt;
        return;
      }
      node = stack[--sp];
    }
  }
  out->n = kCodePerRay;
}

// Mean horizontal spacing of the mesh's triangles: the square root of its area
// over their number.
__device__ __forceinline__ float tri_spacing(const MeshDev& m) {
  float lo[2] = {INFINITY, INFINITY}, hi[2] = {-INFINITY, -INFINITY};
  for (int k = 0; k < 2; ++k) {  // the root's children (an unused one is at 1e30)
    const float4 mn = __ldg(m.nodes + 2 * k), mx = __ldg(m.nodes + 2 * k + 1);
    if (mn.x >= 1e29f) continue;
    lo[0] = fminf(lo[0], mn.x);
    lo[1] = fminf(lo[1], mn.y);
    hi[0] = fmaxf(hi[0], mx.x);
    hi[1] = fmaxf(hi[1], mx.y);
  }
  return sqrtf((hi[0] - lo[0]) * (hi[1] - lo[1]) / (float)m.n_tris);
}

// Mean and spread of the offsets of about kBoxSample particles (exact integer sums,
// so the grid does not depend on the order), then the grid: cubic cells over the
// mean +- 4.2 standard deviations (outside it rays walk by themselves, 30 times the work),
// about n / PF_CELL_PARTICLES within +- 3.2.
__global__ void __launch_bounds__(kThreads) k_cells_box(EngineDev e, int f, MeshDev m, CellGrid* g, int n_sat) {
  const FilterDesc* fd = e.desc + f;
  const FilterCtrl* fc = e.ctrl + f;
  const ParticleSrc ps = particle_src(e, fd, fc);
  long long s1[3] = {0, 0, 0}, s2[3] = {0, 0, 0};
  unsigned cnt = 0;
  const int step = max(1, ps.n / kBoxSample);  // of warps
  for (int i = blockIdx.x * kThreads + threadIdx.x;; i += gridDim.x * kThreads) {
    const long long j = (long long)(i >> 5) * step * 32 + (i & 31);
    if (j >= ps.n) break;
    const float* sp = particle_at(e, ps, (int)j);
    const float x[3] = {__ldcg(sp), __ldcg(sp + e.p_total), __ldcg(sp + 2 * e.p_total)};
    if (!(isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]))) continue;
    ++cnt;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const long long q = __float2int_rn(100.f * fminf(fmaxf(x[a], -2000.f), 2000.f));
      s1[a] += q;
      s2[a] += q * q;
    }
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    s1[a] = (long long)warp_sum_u64((unsigned long long)s1[a]);
    s2[a] = (long long)warp_sum_u64((unsigned long long)s2[a]);
  }
  __shared__ bool s_last;
  __shared__ unsigned long long s_sum[7];
  if (threadIdx.x < 7) s_sum[threadIdx.x] = 0ull;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&s_sum[0], (unsigned long long)cnt);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      atomicAdd(&s_sum[1 + a], (unsigned long long)s1[a]);
      atomicAdd(&s_sum[4 + a], (unsigned long long)s2[a]);
    }
  }
  __syncthreads();
  if (threadIdx.x < 7)
    atomicAdd(threadIdx.x == 0   ? &g->count
              : threadIdx.x <= 3 ? (unsigned long long*)&g->s1[threadIdx.x - 1]
                                 : (unsigned long long*)&g->s2[threadIdx.x - 4],
              s_sum[threadIdx.x]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&g->ticket, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!s_last || threadIdx.x != 0) return;
  __threadfence();
  const double nv = (double)max(1ull, __ldcg(&g->count));
  double mu[3], wid[3];
  for (int a = 0; a < 3; ++a) {
    mu[a] = (double)__ldcg(&g->s1[a]) / nv;
    const double var = fmax(0.0, (double)__ldcg(&g->s2[a]) / nv - mu[a] * mu[a]);
    mu[a] *= 0.01;
    wid[a] = fmax(8.4 * 0.01 * sqrt(var), 0.05);
  }
  const int want = cells_wanted(ps.n, n_sat);
  const int bc[3] = {4, 4, 2};
  float side = (float)cbrt(wid[0] * wid[1] * wid[2] / want);
  int dim[3];
  for (int it = 0;; ++it) {  // rounding the counts up may exceed the cells there are
    long long c = kBlockCells;
    for (int a = 0; a < 3; ++a) {
      dim[a] = max(1, (int)ceil(fmin(wid[a] / (bc[a] * side), 1e6)));
      c *= dim[a];
    }
    if (c <= (long long)want + want / 4) break;
    if (it == 64) {
      dim[0] = dim[1] = dim[2] = 1;
      break;
    }
    side *= 1.1f;
  }
  for (int a = 0; a < 3; ++a) {
    g->bdim[a] = dim[a];
    g->lo[a] = (float)(mu[a] - 0.5 * dim[a] * bc[a] * side);
  }
  g->side = side;
  g->inv_side = 1.0f / side;
  g->n_blocks = side <= kCellSpan * tri_spacing(m) ? dim[0] * dim[1] * dim[2] : 0;
  const double* rf = fd->rot;
  for (int r = 0; r < 3; ++r) {
    double o = 0.0;
    float M[3];
    for (int k = 0; k < 3; ++k) {
      o += m.rot[3 * r + k] * (fc->anchor[k] - m.origin[k]);
      M[k] = (float)(m.rot[3 * r] * rf[3 * k] + m.rot[3 * r + 1] * rf[3 * k + 1] + m.rot[3 * r + 2] * rf[3 * k + 2]);
      g->M[3 * r + k] = M[k];
    }
    g->off[r] = (float)o;
    g->hm[r] = fabsf(M[0]) + fabsf(M[1]) + fabsf(M[2]);
    g->hb[r] = 4.f * fabsf(M[0]) + 4.f * fabsf(M[1]) + 2.f * fabsf(M[2]);
  }
}

// The cell of local offsets x (block x 32 + cell of the block); -1 outside
// the grid.
__device__ __forceinline__ int cell_of(const CellGrid* g, float x0, float x1, float x2) {
  const float inv = g->inv_side;
  const float a = floorf((x0 - g->lo[0]) * inv), b = floorf((x1 - g->lo[1]) * inv), c = floorf((x2 - g->lo[2]) * inv);
  const int d0 = g->bdim[0], d1 = g->bdim[1], d2 = g->bdim[2];
  if (!(a >= 0.f && b >= 0.f && c >= 0.f && a < 4.f * d0 && b < 4.f * d1 && c < 2.f * d2)) return -1;
  const int ia = (int)a, ib = (int)b, ic = (int)c;
  return ((((ic >> 1) * d1 + (ib >> 2)) * d0 + (ia >> 2)) << 5) | ((ic & 1) << 4) | ((ib & 3) << 2) | (ia & 3);
}

// Mesh-frame point of local offsets.
__device__ __forceinline__ float3 grid_point(const CellGrid* g, float x, float y, float z) {
  return make_float3(g->M[0] * x + g->M[1] * y + g->M[2] * z + g->off[0],
                     g->M[3] * x + g->M[4] * y + g->M[5] * z + g->off[1],
                     g->M[6] * x + g->M[7] * y + g->M[8] * z + g->off[2]);
}

__global__ void __launch_bounds__(kThreads) k_cells_mark(EngineDev e, int f, CellBufs cb) {
  __shared__ unsigned s_bits[kCellsMax / kBlockCells / 32 + 1];  // marks collected per CTA: few words, many writers
  const ParticleSrc ps = particle_src(e, e.desc + f, e.ctrl + f);
  const int words = (cb.grid->n_blocks + 31) / 32;
  if (words == 0) return;
  for (int i = threadIdx.x; i < words; i += kThreads) s_bits[i] = 0u;
  __syncthreads();
  for (int j = blockIdx.x * kThreads + threadIdx.x; j < ps.n; j += gridDim.x * kThreads) {
    const float* sp = particle_at(e, ps, j);
    const int c = cell_of(cb.grid, __ldcg(sp), __ldcg(sp + e.p_total), __ldcg(sp + 2 * e.p_total));
    if (c < 0) continue;
    const unsigned bit = 1u << ((c >> 5) & 31);
    if (!(*(volatile unsigned*)&s_bits[c >> 10] & bit)) atomicOr(&s_bits[c >> 10], bit);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < words; i += kThreads)
    if (s_bits[i] & ~__ldcg(cb.mark + i)) atomicOr(cb.mark + i, s_bits[i]);
}
__device__ __forceinline__ bool marked(const CellBufs& cb, int b) { return (cb.mark[b >> 5] >> (b & 31)) & 1u; }

// One thread per (satellite, block), blocks fastest: a warp walks with
// neighbouring blocks to one satellite, along nearly one path.
__global__ void __launch_bounds__(128) k_cells_block(MeshDev m, const Sat3d* sats, int n_sat, CellBufs cb) {
  const CellGrid* g = cb.grid;
  const int nb = g->n_blocks;
  const float side = g->side, half = 0.5f * side * 1.001f + 1e-4f;
  const float3 h = make_float3(g->hb[0] * half, g->hb[1] * half, g->hb[2] * half);
  for (int i = blockIdx.x * 128 + threadIdx.x; i < nb * n_sat; i += gridDim.x * 128) {
    const int s = i / nb, b = i - s * nb;
    if (!marked(cb, b)) continue;
    const int d0 = g->bdim[0], d1 = g->bdim[1];
    const float3 c = grid_point(g, g->lo[0] + (4.f * (float)(b % d0) + 2.f) * side,
                                g->lo[1] + (4.f * (float)(b / d0 % d1) + 2.f) * side,
                                g->lo[2] + (2.f * (float)(b / (d0 * d1)) + 1.f) * side);
    beam_walk(m, c, h, mesh_origin(m, sats[s].sat), cb.list + (size_t)b * n_sat + s);
  }
}

// One warp per (block, satellite), one lane per cell.
__global__ void __launch_bounds__(kThreads) k_cells_cell(MeshDev m, const Sat3d* sats, int n_sat, CellBufs cb) {
  const CellGrid* g = cb.grid;
  const int lane = threadIdx.x & 31, warps = gridDim.x * (kThreads / 32);
  const float side = g->side, half = 0.5f * side * 1.001f + 1e-4f;
  const float3 h = make_float3(g->hm[0] * half, g->hm[1] * half, g->hm[2] * half);
  for (int i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); i < g->n_blocks * n_sat; i += warps) {
    const int b = i / n_sat, s = i - b * n_sat;
    if (!marked(cb, b)) continue;
    const BlockList* bl = cb.list + i;
    const unsigned n = bl->n;
    unsigned code = n;
    if (n <= (unsigned)kBeamCap) {
      code = 0u;
      if (n > 0u) {
        const int d0 = g->bdim[0], d1 = g->bdim[1];
        const float3 c = grid_point(g, g->lo[0] + (float)(4 * (b % d0) + (lane & 3)) * side + 0.5f * side,
                                    g->lo[1] + (float)(4 * (b / d0 % d1) + ((lane >> 2) & 3)) * side + 0.5f * side,
                                    g->lo[2] + (float)(2 * (b / (d0 * d1)) + (lane >> 4)) * side + 0.5f * side);
        const float3 sat = mesh_origin(m, sats[s].sat);
        const Beam beam = make_beam(c, h, sat, dist3(sat, c), bl->ext);
        for (unsigned q = 0; q < n; ++q) {
          const float4* t = m.tris + 3 * bl->tri[q];
          const int r = beam_triangle(beam, __ldg(t), __ldg(t + 1), __ldg(t + 2));
          if (r == 2) code = kCodeBlocked;
          else if (r == 1 && code != kCodeBlocked) code |= 1u << q;
          if (__all_sync(0xffffffffu, code == kCodeBlocked)) break;
        }
      }
    }
    cb.code[((size_t)b * kBlockCells + lane) * n_sat + s] = code;
  }
}

// One thread per ray: a warp takes one satellite and 32 particles in a row.
__global__ void __launch_bounds__(kThreads) k_rays_3d(EngineDev e, int f, MeshDev m, const Sat3d* sats, int n_sat,
                                                      unsigned* blk) {
  const FilterDesc* fd = e.desc + f;
  const FilterCtrl* fc = e.ctrl + f;
  const ParticleSrc ps = particle_src(e, fd, fc);
  const int lane = threadIdx.x & 31, words = (ps.n + 31) / 32, warps = gridDim.x * (kThreads / 32);
  for (int i = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); i < words * n_sat; i += warps) {
    const int s = i / words, j = (i - s * words) * 32 + lane;
    const float* sp = particle_at(e, ps, min(j, ps.n - 1));
    double p[3];
    local_to_ecef(fd->rot, fc->anchor, (double)__ldcg(sp), (double)__ldcg(sp + e.p_total),
                  (double)__ldcg(sp + 2 * e.p_total), p);
    const double v[3] = {sats[s].sat[0] - p[0], sats[s].sat[1] - p[1], sats[s].sat[2] - p[2]};
    const double L = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    const unsigned w = __ballot_sync(0xffffffffu, bvh_blocked(m, mesh_origin(m, p), mesh_dir(m, v, L), (float)L));
    if (lane == 0) blk[i] = w;
  }
}

// Satellite and NLOS terms of one particle, with its rays' verdicts from its
// own walks (RAYS_WALK), from the words of k_rays_3d, or from its cell (and its
// own rays where the cells left them open).  One particle per thread.
template <int MODE>
__global__ void __launch_bounds__(kThreads, MODE == RAYS_CELLS ? 3 : 4) k_weight_3d(EngineDev e, int f, MeshDev m,
                                                                                   const Sat3d* sats, Weight3dArgs a,
                                                                                   CellBufs cb) {
  constexpr int kWarps = kThreads / 32, kQueue = 64;
  constexpr int kSlots = MODE == RAYS_CELLS ? kWarps : 1;  // the queues are the cells'
  // with a grid, its kernel and the walking one are both launched: the cloud decides
  if (MODE == RAYS_CELLS && cb.grid->n_blocks == 0) return;
  if (MODE == RAYS_WALK && cb.grid && cb.grid->n_blocks != 0) return;
  __shared__ Sat3d s_sat[kMax3dSats];
  __shared__ double s_p[kSlots][3][32];
  __shared__ unsigned long long s_blk[kSlots][32];
  __shared__ unsigned s_code[kSlots][kQueue];
  __shared__ unsigned short s_item[kSlots][2][kQueue];
  __shared__ int s_block[kSlots][32];
  for (int i = threadIdx.x; i < a.n_sat; i += kThreads) s_sat[i] = sats[i];
  __syncthreads();
  const FilterDesc* fd = e.desc + f;
  const FilterCtrl* fc = e.ctrl + f;
  const ParticleSrc ps = particle_src(e, fd, fc);
  const int n = ps.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long base = ps.base;
  const bool keep = a.accumulate && fc->lw_zero == 0;
  for (int j0 = (blockIdx.x * kThreads + threadIdx.x) & ~31; j0 < n; j0 += gridDim.x * kThreads) {
    const int j = j0 + lane;
    const bool in = j < n;
    const float* sp = particle_at(e, ps, in ? j : n - 1);
    const float x0 = __ldcg(sp), x1 = __ldcg(sp + e.p_total), x2 = __ldcg(sp + 2 * e.p_total),
                x3 = __ldcg(sp + 3 * e.p_total);
    double p[3];
    local_to_ecef(fd->rot, fc->anchor, (double)x0, (double)x1, (double)x2, p);
    const double clk = fc->clk_anchor[0] + (double)x3;
    unsigned long long blk = 0ull;
    if constexpr (MODE == RAYS_WORDS)
      for (int s = 0; s < a.n_sat; ++s)
        blk |= (unsigned long long)((__ldcg(cb.blk + (size_t)s * ((n + 31) / 32) + j0 / 32) >> lane) & 1u) << s;
    if constexpr (MODE == RAYS_CELLS) {
      const int cell = cell_of(cb.grid, x0, x1, x2);
      s_blk[warp][lane] = 0ull;
      s_block[warp][lane] = cell >> 5;
#pragma unroll
      for (int q = 0; q < 3; ++q) s_p[warp][q][lane] = p[q];
      __syncwarp();
      // open rays are queued and tested by whole warps: queue 0 those with a
      // list, queue 1 those that walk the hierarchy (much longer)
      int queued[2] = {0, 0};
      auto drain = [&](int which, int count) {
        if (lane < count) {
          const int own = s_item[warp][which][lane] & 31, s = s_item[warp][which][lane] >> 5;
          const Sat3d& sv = s_sat[s];
          const double pq[3] = {s_p[warp][0][own], s_p[warp][1][own], s_p[warp][2][own]};
          const double v[3] = {sv.sat[0] - pq[0], sv.sat[1] - pq[1], sv.sat[2] - pq[2]};
          const double L = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
          const float3 o = mesh_origin(m, pq), d = mesh_dir(m, v, L);
          bool hit = false;
          if (which) {
            hit = bvh_blocked(m, o, d, (float)L);
          } else {
            const int* list = cb.list[(size_t)s_block[warp][own] * a.n_sat + s].tri;
            for (unsigned left = s_code[warp][lane]; left && !hit; left &= left - 1u) {
              const float4* t = m.tris + 3 * list[__ffs(left) - 1];
              hit = tri_hit(o, d, __ldg(t), __ldg(t + 1), __ldg(t + 2), (float)L);
            }
          }
          if (hit) atomicOr(&s_blk[warp][own], 1ull << s);
        }
      };
#pragma unroll 1
      for (int s0 = 0; s0 < a.n_sat; s0 += 4) {
        unsigned code4[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          code4[q] = s0 + q >= a.n_sat ? 0u
                     : cell >= 0 ? __ldcg(cb.code + (size_t)cell * a.n_sat + s0 + q)
                                 : kCodePerRay;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const unsigned code = code4[q];
          if (code == kCodeBlocked) blk |= 1ull << (s0 + q);
          const bool open = code != 0u && code != kCodeBlocked;
          if (!__any_sync(0xffffffffu, open)) continue;
#pragma unroll
          for (int which = 0; which < 2; ++which) {
            const bool mine = open && (code == kCodePerRay) == (which == 1);
            const unsigned mask = __ballot_sync(0xffffffffu, mine);
            if (!mask) continue;
            if (mine) {
              const int at = queued[which] + __popc(mask & ((1u << lane) - 1u));
              s_item[warp][which][at] = (unsigned short)(((s0 + q) << 5) | lane);
              if (which == 0) s_code[warp][at] = code;
            }
            queued[which] += __popc(mask);
            __syncwarp();
            if (queued[which] >= 32) {
              drain(which, 32);
              queued[which] -= 32;
              __syncwarp();
              if (lane < queued[which]) {  // the rest moves to the front
                s_item[warp][which][lane] = s_item[warp][which][32 + lane];
                if (which == 0) s_code[warp][lane] = s_code[warp][32 + lane];
              }
              __syncwarp();
            }
          }
        }
      }
      drain(0, queued[0]);
      drain(1, queued[1]);
      __syncwarp();
      blk |= s_blk[warp][lane];
    }
    const float3 o = MODE == RAYS_WALK ? mesh_origin(m, p) : make_float3(0.f, 0.f, 0.f);
    double acc = 0.0;
#pragma unroll 1
    for (int s = 0; s < a.n_sat; ++s) {
      const Sat3d& sv = s_sat[s];
      const double v[3] = {sv.sat[0] - p[0], sv.sat[1] - p[1], sv.sat[2] - p[2]};
      const double L = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
      const bool hit = MODE == RAYS_WALK ? bvh_blocked(m, o, mesh_dir(m, v, L), (float)L) : ((blk >> s) & 1ull) != 0ull;
      const double r = sv.pr - (L + clk);
      const double los = -0.5 * sv.w * r * r * a.inv_s2_los;
      const double rn = r > 0.0 ? r - a.nlos_bias : r;
      const double nlos = -0.5 * sv.w * rn * rn * a.inv_s2_nlos;
      acc += mix_loglik(los, nlos, hit ? a.p_blocked : a.p_clear);
    }
    if (in) {
      const float l0 = keep ? e.lw[base + j] : 0.f;
      e.lw[base + j] = (float)((double)l0 + acc);
    }
    __syncwarp();
  }
}

// Line of sight of n_ray rays: receiver rx[i / n_sat] to satellite
// sat[i] (ECEF, FP64); los[i] = 1 when clear.  Non-finite inputs give 0.
__global__ void __launch_bounds__(kThreads) k_bvh_los(MeshDev m, const double* rx, const double* sat, int n_rx,
                                                      int n_sat, unsigned char* los) {
  const long long total = (long long)n_rx * n_sat;
  for (long long i = blockIdx.x * (long long)kThreads + threadIdx.x; i < total; i += (long long)gridDim.x * kThreads) {
    const long long r = i / n_sat;
    const double p[3] = {rx[3 * r], rx[3 * r + 1], rx[3 * r + 2]};
    const double s[3] = {sat[3 * i], sat[3 * i + 1], sat[3 * i + 2]};
    bool ok = true;
    for (int a = 0; a < 3; ++a) ok = ok && isfinite(p[a]) && isfinite(s[a]);
    if (!ok) {
      los[i] = 0;
      continue;
    }
    const double v[3] = {s[0] - p[0], s[1] - p[1], s[2] - p[2]};
    const double L = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    los[i] = bvh_blocked(m, mesh_origin(m, p), mesh_dir(m, v, L), (float)L) ? 0 : 1;
  }
}

}  // namespace pfb
