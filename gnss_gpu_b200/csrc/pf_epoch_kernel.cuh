// pf_epoch_kernel.cuh -- one cooperative persistent kernel per epoch.
//
// All CTAs are co-resident (cooperative launch); each owns a contiguous
// chunk of (filter, tile) work items and the phases of the epoch are
// separated by one grid barrier with bounded spins:
//
//   1  predict + likelihood + tile statistics (particles loaded straight
//      into registers, gathered through the last resample's ancestors;
//      measured faster than staging them through shared memory with
//      cp.async).  Systematic: also the segment and tile levels of the
//      tiled integer CDF -- each warp quantises its 128 particles against
//      its own maximum and stores their prefixes inside the segment, and the
//      warp that merges the tile's rows (the warps take turns, two tiles
//      behind) rescales the segment sums exactly to the tile maximum.
//   -- barrier
//   2  per-filter merge of the tile rows (filter f_first + j by CTA j mod G):
//      ESS, weighted mean / covariance, device-side resample decision.
//      At the same time, systematic only, on the CTAs that own no filter
//      (when filters are fewer than a quarter of the CTAs; otherwise every
//      CTA after its merges):
//   4  the filter maximum from the tile maxima, tile sums rescaled to it,
//      the filter prefix of each tile, then per particle its filter-wide CDF
//      and offspring end F(i); slots [F(i-1), F(i)) get ancestor i, written
//      by the lane when the run is short and by the warp when it is long,
//      where a 128-slot segment the run covers gets one marker word instead
//      of 128 slots (speculative for every filter that may resample: the
//      decision is taken meanwhile).  The kernel ends there.
//   Megopolis instead: every CTA takes the resample decision for the
//   filters of its tiles from the owner's merge (recomputed, bit-identical),
//   then runs the chain per slot of its tiles.  The kernel ends there.
//
// Compared with one kernel per phase this removes the launch/drain gaps and
// every per-tile queue atomic; the prefixes reread in phase 4 come from L2
// (the epoch just wrote them).  Phase 4 needs no CTA barrier per tile: warps
// work on independent segments.
#pragma once
#include <type_traits>

#include "pf_engine_kernels.cuh"
#include "pf_learned.cuh"
#include "pf_generic.cuh"

namespace pfb {

__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Grid barrier for co-resident CTAs (sense reversal on one arrival counter).
// bar[1] is the generation (the count of barriers passed over all launches),
// bar[kBarCount] the arrivals at the current barrier; `gen` is this CTA's
// copy of the generation.  Thread 0 of every CTA adds its arrival with one
// acquire-release atomic (the release publishes the writes its CTA ordered
// before it with __syncthreads); the CTA that arrives last resets the
// counter and releases the grid with one store of the next generation,
// which the others poll (relaxed loads, then one fence).  One hop from the
// last arrival to the release: measured 1.6-3.1 us per barrier at 296 CTAs
// against 2.8-5.1 us for per-CTA arrival flags collected by CTA 0.  Waits
// are bounded: on timeout the error word is set and the CTA goes on (results
// are then invalid, and the host reports PF_ETIMEOUT).
__device__ __forceinline__ void grid_barrier(const EngineDev& e, unsigned* bar, unsigned& gen) {
  const unsigned target = gen + 1u;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(bar + kBarCount) : "memory");
    if (old == gridDim.x - 1u) {  // the last CTA to arrive releases the grid
      bar[kBarCount] = 0u;
      st_release(bar + 1, target);
    }
    const unsigned want = e.lookback_poison ? target + 1u : target;
    unsigned long long spins = 0;
    while (ld_relaxed(bar + 1) != want) {
      if (++spins > e.spin_limit) {
        raise_err(e, ERR_BARRIER_TIMEOUT);
        break;
      }
      if (spins > 64) __nanosleep(32);
    }
    fence_acq_rel();
  }
  gen = target;
  __syncthreads();
}

// Hand-over of the warps' statistics rows to the warp that merges a tile
// (shared-memory counters, release / acquire at CTA scope).
__device__ __forceinline__ void cta_red_release(unsigned* p) {
  asm volatile("red.release.cta.shared.add.u32 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void cta_st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}
// Waits until *p has reached `want` (counters only grow).  The other warps of
// the CTA always run on, so the wait ends; the limit only guards against a
// fault elsewhere.
__device__ __forceinline__ void cta_wait_reach(const EngineDev& e, const unsigned* p, unsigned want) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  for (unsigned spins = 0;; ++spins) {
    unsigned v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    if ((int)(v - want) >= 0) return;
    if (spins > (1u << 24)) {
      raise_err(e, ERR_BARRIER_TIMEOUT);
      return;
    }
  }
}

// Reads through L2 of control-block fields that another CTA wrote before a
// grid barrier (L1 is not coherent across SMs).
__device__ __forceinline__ int ld_cg_int(const int* p) { return __ldcg(p); }
__device__ __forceinline__ unsigned ld_cg_u(const unsigned* p) { return __ldcg(p); }
__device__ __forceinline__ float ld_cg_f(const float* p) { return __ldcg(p); }

// Chunk of worker w out of nw over the work items [t0, t0 + count).
__device__ __forceinline__ void chunk_of(int t0, int count, int w, int nw, int& b, int& e) {
  const int per = count / nw, rem = count % nw;
  b = t0 + w * per + min(w, rem);
  e = b + per + (w < rem ? 1 : 0);
}
__device__ __forceinline__ void cta_chunk(int t0, int count, int& b, int& e) {
  chunk_of(t0, count, (int)blockIdx.x, (int)gridDim.x, b, e);
}

// Phase 1's chunk of this CTA.  With many filters a tile's cost depends on its
// filter's satellites, so the tiles are cut by cost, not by number: a tile
// costs kFix + n_sat in units of one satellite, and CTA w takes the tiles whose
// starts lie in [w, w + 1) / G of the whole cost.  kFix is the rest of a tile
// (draws, statistics, CDF) over one satellite, fitted to phase 1 of 48 x 100K
// filters with 8 to 40 satellites (per tile, one clock, us: Gaussian 4.3 + 0.084
// s, Huber 4.1 + 0.114 s, mixture 4.4 + 0.27 s).  256 filters with 6 to 40
// satellites: phase 1 ended between 88 and 178 us with equal numbers.  With several
// clocks the same times 8 / 5, chosen between 5 / 5 and 12 / 5 (256 x 20K Huber filters
// of 4 clocks 248 us; 260 and 249 us; the Gaussian ones 213; 215 and 217).
//
// The cut itself is three dependent loads per filter and a scan, 3 us for 256
// filters, 8 for 1024 and 40 for 4096, and a chunk of many small filters has about
// the average satellites anyway: below kCutTiles tiles per filter the numbers are
// equal.  Epoch kernel, us, cut by cost / by number: Huber, 6 to 40 satellites,
// 64 x 15 tiles 56 / 64, 256 x 20 204 / 225, 256 x 10 116 / 123, 1024 x 12 471 / 492,
// 1024 x 6 266 / 267 (Gaussian 224 / 222, mixture 351 / 363), 1024 x 3 167 / 163,
// 256 x 5 70 / 72 (Gaussian 64 / 62, mixture 97 / 94), 4096 x 1 227 / 183; with
// satellites equal throughout the cut costs up to 3 % of the kernel (64 x 30 tiles
// 106 / 102).
constexpr int kCutTiles = 8;
template <int NCLK, int WMODE>
__device__ __forceinline__ void weighted_chunk(const EngineDev& e, int t0, int count, const unsigned char* obs0,
                                               unsigned long long* s_u64, int* s_cut, int& cb, int& ce) {
  constexpr int kFix = (WMODE == PF_WEIGHT_GAUSSIAN ? 48 : WMODE == PF_WEIGHT_MIXTURE ? 22 : 34) * (NCLK > 1 ? 8 : 5) / 5;
  const int f0 = __ldg(e.tile_filter + t0), nf = __ldg(e.tile_filter + t0 + count - 1) - f0 + 1;
  if (count <= (int)gridDim.x || nf == 1 || count < kCutTiles * nf) {  // CTA-uniform; the first needs no load
    cta_chunk(t0, count, cb, ce);
    return;
  }
  const int per = (nf + kThreads - 1) / kThreads, a = min((int)threadIdx.x * per, nf), b = min(a + per, nf);
  auto tiles_of = [&](int f) {  // of the launch
    const FilterDesc* fd = e.desc + f;
    return min(fd->tile_begin + fd->n_tiles, t0 + count) - max(fd->tile_begin, t0);
  };
  auto cost_of = [&](int f) {
    const unsigned epoch = e.ctrl[f].epoch;
    const pf_filter_epoch_t* fe =
        reinterpret_cast<const pf_filter_epoch_t*>(obs0 + (size_t)(epoch % (unsigned)e.obs_slots) * e.obs_slot_bytes) + f;
    return (unsigned long long)(kFix + ((fe->flags & PF_EP_WEIGHT) ? min(max(fe->n_sat, 0), e.max_sats) : 0));
  };
  unsigned long long mine = 0, total;
  for (int k = a; k < b; ++k) mine += cost_of(f0 + k) * (unsigned long long)tiles_of(f0 + k);
  if (threadIdx.x < 2) s_cut[threadIdx.x] = 0;
  unsigned long long at = block_excl_scan_u64(mine, s_u64, &total);
  // tiles that start below each end of the CTA's share
  const unsigned long long lo = total * blockIdx.x / gridDim.x, hi = total * (blockIdx.x + 1ull) / gridDim.x;
  int n_lo = 0, n_hi = 0;
  for (int k = a; k < b; ++k) {
    const unsigned long long c = cost_of(f0 + k), nt = (unsigned long long)tiles_of(f0 + k);
    if (lo > at) n_lo += (int)min(nt, (lo - at + c - 1) / c);
    if (hi > at) n_hi += (int)min(nt, (hi - at + c - 1) / c);
    at += c * nt;
  }
  n_lo = __reduce_add_sync(0xffffffffu, n_lo);
  n_hi = __reduce_add_sync(0xffffffffu, n_hi);
  if ((threadIdx.x & 31) == 0) {  // s_cut was cleared before the scan's barriers
    if (n_lo) atomicAdd(s_cut, n_lo);
    if (n_hi) atomicAdd(s_cut + 1, n_hi);
  }
  __syncthreads();
  cb = t0 + s_cut[0];
  ce = t0 + s_cut[1];
}

// Block-wide sums of two 64-bit values (s_tmp: 2 * kWarps words).
__device__ __forceinline__ void block_sum2_u64(unsigned long long a, unsigned long long b,
                                               unsigned long long* s_tmp, unsigned long long& ra,
                                               unsigned long long& rb) {
  constexpr int kWarps = kThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  a = warp_sum_u64(a);
  b = warp_sum_u64(b);
  __syncthreads();
  if (lane == 0) {
    s_tmp[warp] = a;
    s_tmp[kWarps + warp] = b;
  }
  __syncthreads();
  ra = 0ull;
  rb = 0ull;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    ra += s_tmp[w];
    rb += s_tmp[kWarps + w];
  }
}


// The systematic resampler's phase 4 walks a chunk of tiles filter segment
// by filter segment (the tiles of one filter inside the chunk).  Every warp
// works on its own 128-particle segment without CTA barriers; only the
// per-filter maximum and prefix are CTA reductions.  The loops are kept
// compact (not unrolled over tiles): this code runs a few times per CTA and
// epoch, so instruction fetch, not arithmetic, sets its speed.  Integer sums
// are exact, so the result does not depend on the chunking.

// Phase 4's inputs of one tile for one lane: the tile's integer sum and
// maximum, its warp segment's scale and prefix, the lane's four in-segment
// prefixes (zero past the filter's end).
struct OffspringTileIn {
  double S, rho, E;
  double2 ca, cb;
  float m;
};
__device__ __forceinline__ OffspringTileIn load_offspring_tile(const EngineDev& e, int g, int tb, int n,
                                                               long long base, int warp, int lane) {
  OffspringTileIn o;
  o.S = __ldcg(e.tile_S + g);
  o.m = __ldcg(e.tile_m + g);
  o.rho = 0.0;
  o.E = 0.0;
  o.ca = make_double2(0.0, 0.0);
  o.cb = o.ca;
  const int pw = (g - tb) * kTile + warp * kWarpTile, p0 = pw + lane * 4;
  if (pw < n) {
    o.rho = __ldcg(e.seg_rho + (size_t)g * kSubTiles + warp);
    o.E = __ldcg(e.seg_E + (size_t)g * kSubTiles + warp);
    if (p0 < n) {
      const double2* src = reinterpret_cast<const double2*>(e.seg_c + base + p0);
      o.ca = __ldcg(src);
      o.cb = __ldcg(src + 1);
    }
  }
  return o;
}

// The run [lo, hi) of ancestor i, written by the whole warp (its values
// broadcast from one lane): the marker of every 128-slot segment that starts
// inside the run -- i when the run covers the segment, else -1 (only the
// last one can be partial) -- and the slots of the segments the run covers
// in part.  `seg` is the filter's marker array, n its slot count.
__device__ __forceinline__ void write_heavy_run(const EngineDev& e, int* anc, int* seg, uint32_t lo, uint32_t hi,
                                                int i, uint32_t n, int lane) {
  if (!PF_BOUNDS_OK(e, lo < hi && hi <= n)) return;
  const uint32_t s_first = (lo + kWarpTile - 1) / kWarpTile, s_last = (hi - 1) / kWarpTile;
  const bool last_full = s_first <= s_last && min((s_last + 1) * (uint32_t)kWarpTile, n) <= hi;
  for (uint32_t sg = s_first + lane; sg <= s_last; sg += 32) seg[sg] = (sg < s_last || last_full) ? i : -1;
  const uint32_t head_end = min(hi, s_first * (uint32_t)kWarpTile);
  for (uint32_t j = lo + lane; j < head_end; j += 32) anc[j] = i;
  if (s_first <= s_last && !last_full)
    for (uint32_t j = s_last * (uint32_t)kWarpTile + lane; j < hi; j += 32) anc[j] = i;
}

// Phase 4, right after the grid barrier and speculative (the filters'
// owners decide at the same time whether they resample; when one does not,
// this work is unused): for every filter that may resample this step (the
// flag phase 1 left in its control block), the filter maximum from the tile
// maxima, the filter prefix of each tile of the chunk from the tile sums
// scaled to that maximum, then per particle its filter-wide CDF C_i and
// offspring end F(i); slots [F(i-1), F(i)) get ancestor i.  A run of up to
// kLightRun slots is written by its lane (with the marker of a segment
// starting inside it); a longer one by the whole warp (write_heavy_run).
// The marker of each segment is written by the run holding the segment's
// first slot, so every resampling step rewrites all of them, and the step
// needs no second grid barrier: the next step's gather is the first reader.
__device__ __forceinline__ void epoch_sys_offspring(const EngineDev& e, int cb, int ce, unsigned long long* s_u64) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t = cb; t < ce;) {
    const int f = __ldg(e.tile_filter + t);
    const FilterDesc* fd = e.desc + f;
    FilterCtrl* fc = e.ctrl + f;
    const int tb = fd->tile_begin, nt = fd->n_tiles, se = min(ce, tb + nt);
    if (ld_cg_int(&fc->sys_q_cur)) {  // CTA-uniform
      const int n = fd->n;
      const long long base = fd->p_off;
      // the first tile's inputs load while the filter prefix is formed; in
      // the loop below the next tile's load while this one is worked on
      // (every load is independent of the previous tile)
      OffspringTileIn nxt{};
      if (t < se) nxt = load_offspring_tile(e, t, tb, n, base, warp, lane);
      // the filter maximum M (the largest tile maximum), then the prefix of
      // tile t inside its filter and the filter total, from the tile sums
      // scaled to M; four tiles per thread and round, their loads issued
      // together, one round kept in registers for filters of up to
      // kB * kThreads tiles
      constexpr int kB = 4;
      double S[kB];
      float m[kB];
      auto load_round = [&](int i0) {
#pragma unroll
        for (int j = 0; j < kB; ++j) {
          const int i = i0 + j * kThreads;
          S[j] = i < nt ? __ldcg(e.tile_S + tb + i) : 0.0;
          m[j] = i < nt ? __ldcg(e.tile_m + tb + i) : -INFINITY;
        }
      };
      float mx = -INFINITY;
#pragma unroll 1
      for (int i0 = threadIdx.x; i0 < nt; i0 += kB * kThreads) {
        load_round(i0);
#pragma unroll
        for (int j = 0; j < kB; ++j) mx = fmaxf(mx, m[j]);
      }
      const float M = block_max(mx, reinterpret_cast<float*>(s_u64));
      if (M == -INFINITY) {  // CTA-uniform: no finite weight (the owner reports it)
        t = se;
        continue;
      }
      unsigned long long P = 0, W = 0;
      {
        unsigned long long pre = 0, all = 0;
#pragma unroll 1
        for (int i0 = threadIdx.x; i0 < nt; i0 += kB * kThreads) {
          if (nt > kB * kThreads) load_round(i0);  // else the registers hold the only round
#pragma unroll
          for (int j = 0; j < kB; ++j) {
            double r;
            const unsigned long long v = (unsigned long long)sys_tile_total(S[j], m[j], M, r);
            all += v;
            if (tb + i0 + j * kThreads < t) pre += v;
          }
        }
        block_sum2_u64(pre, all, s_u64, P, W);
      }
      if (threadIdx.x == 0) {
        if (se == tb + nt) fc->wq_total = W;  // the chunk holding the filter's last tile
        if (W == 0ull) raise_err(e, ERR_BAD_WEIGHTS);
      }
      if (W > 0ull) {
        const uint32_t u = ld_cg_u(&fc->sys_u_cur);
        const double scale = (double)n / (double)W, uf = (double)u * 2.3283064365386963e-10;
        int* anc = e.anc + base;
        int* seg = e.seg_anc + (size_t)tb * kSubTiles;
#pragma unroll 1
        for (int g = t; g < se; ++g) {
          const int pw = (g - tb) * kTile + warp * kWarpTile;
          const int p0 = pw + lane * 4;
          const OffspringTileIn cur = nxt;
          if (g + 1 < se) nxt = load_offspring_tile(e, g + 1, tb, n, base, warp, lane);
          double r;
          const unsigned long long ts = (unsigned long long)sys_tile_total(cur.S, cur.m, M, r);
          if (pw < n) {  // warp-uniform
            const double rho = cur.rho, E = cur.E;
            // segment prefixes of this lane's particles and of the one before
            const double c[4] = {cur.ca.x, cur.ca.y, cur.cb.x, cur.cb.y};
            double cprev = __shfl_up_sync(0xffffffffu, c[3], 1);
            if (lane == 0) cprev = 0.0;
            const double Pd = (double)P;
            uint32_t Fprev = 0u, Fk[4] = {0u, 0u, 0u, 0u};
            if (p0 < n) {
              Fprev = (p0 == 0) ? 0u
                                : offspring_end_split(P, Pd, sys_inner(E, rho, r, cprev), W, (uint32_t)n, u, scale, uf);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                Fk[k] = (p0 + k < n)
                            ? offspring_end_split(P, Pd, sys_inner(E, rho, r, c[k]), W, (uint32_t)n, u, scale, uf)
                            : (uint32_t)n;
            }
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
              const uint32_t lo = (k == 0) ? Fprev : Fk[k - 1], hi = Fk[k];
              const int i = p0 + k;
              const bool run = i < n && hi > lo;
              const bool heavy = run && hi - lo > (uint32_t)kLightRun;
              if (run && !heavy && PF_BOUNDS_OK(e, hi <= (uint32_t)n)) {
                for (uint32_t j = lo; j < hi; ++j) anc[j] = i;
                const uint32_t sg = (lo + kWarpTile - 1) / kWarpTile;  // a segment starting inside the run
                if (sg * (uint32_t)kWarpTile < hi)
                  seg[sg] = min((sg + 1) * (uint32_t)kWarpTile, (uint32_t)n) <= hi ? i : -1;
              }
              unsigned todo = __ballot_sync(0xffffffffu, heavy);
              while (todo) {  // warp-uniform
                const int src = __ffs(todo) - 1;
                todo &= todo - 1u;
                write_heavy_run(e, anc, seg, __shfl_sync(0xffffffffu, lo, src), __shfl_sync(0xffffffffu, hi, src),
                                pw + src * 4 + k, (uint32_t)n, lane);
              }
            }
          }
          P += ts;
        }
      }
    }
    t = se;
  }
}

// One warp merges the warp rows of tile t (the CTA's j-th) into the tile row
// and, when the filter may resample, forms the tile level of its tiled
// integer CDF.  The order of the sums is fixed, so the merging warp does not
// matter.
constexpr int kRowBufs = 4;   // row buffers
constexpr int kMergeLag = 2;  // tiles between writing and merging the rows
template <int NV, int NW>
__device__ __forceinline__ void merge_rows(const EngineDev& e, int t, int j, const float (*s_wrow)[NW][17],
                                           const double (*s_wq)[NW], const unsigned* s_rows, unsigned* s_merged) {
  const int lane = threadIdx.x & 31, b = j % kRowBufs;
  cta_wait_reach(e, s_rows + b, (unsigned)(NW * (j / kRowBufs + 1)));
  const float (*wr)[17] = s_wrow[b];
  const float mw = lane < NW ? wr[lane][0] : -INFINITY;
  const float tm = warp_max(mw);
  float acc = 0.f;
  if (lane < NV && tm > -INFINITY) {
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float m = wr[w][0];
      if (m > -INFINITY) {
        float sc = exp2f((m - tm) * 1.4426950408889634f);
        if (lane == 1) sc *= sc;
        acc = fmaf(sc, wr[w][1 + lane], acc);
      }
    }
  }
  float* row = e.part + (size_t)t * kPartStride;
  if (lane < NV) row[1 + lane] = acc;
  if (lane == 0) row[0] = tm;
  const double S = lane < NW ? s_wq[b][lane] : 0.0;
  if (__shfl_sync(0xffffffffu, S, 0) >= 0.0) sys_tile_scale(e, t, S, mw, tm);
  __syncwarp();
  if (lane == 0) cta_st_release(s_merged + b, (unsigned)(j / kRowBufs + 1));
}

#ifndef PF_EPOCH_MINB
#define PF_EPOCH_MINB 2  // resident CTAs per SM the epoch kernel is compiled for
#endif
template <int NCLK, int WMODE, int RESAMPLER, class IN>
__global__ void __launch_bounds__(kThreads, PF_EPOCH_MINB) k_epoch(EngineDev e, int t0, int count, unsigned* bar,
                                                                     const __grid_constant__ IN in) {
  constexpr int D = 3 + NCLK;
  constexpr int NV = 2 + D + 6;
  constexpr int kWarps = kThreads / 32;
  constexpr int kStride = (WMODE == PF_WEIGHT_MIXTURE || WMODE == PF_WEIGHT_GENERIC) ? kMixStride : kSatStride;
  __shared__ __align__(16) float2 s_sat[kStride * PF_MAX_SATS];
  __shared__ int s_grp[PF_MAX_CLK + 1];
  __shared__ unsigned char s_clk[PF_MAX_SATS];
  __shared__ float s_wrow[kRowBufs][kWarps][17];
  __shared__ float s_maxtmp[kWarps];
  __shared__ double s_dred[kWarps * 16];
  __shared__ unsigned long long s_u64[2 * kWarps];
  __shared__ double s_wq[kRowBufs][kWarps];  // per-warp sums of the tiled integer CDF
  __shared__ unsigned s_rows[kRowBufs], s_merged[kRowBufs];  // rows written, tiles merged (counts per buffer)
  __shared__ int s_cut[2];
  __shared__ int s_dec_f, s_dec_rs;  // the filter this CTA owns in phase 2 and its decision

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // generation of the last barrier (every thread reads it before its CTA
  // first arrives, so no CTA can have moved it on yet).  A relaxed load: the
  // kernel boundary already orders the previous launch's release, and an
  // acquire here would hold every later load of the CTA behind it.
  unsigned gen = ld_relaxed(bar + 1);
  if (threadIdx.x == 0) s_dec_f = -1;
  if (threadIdx.x < kRowBufs) s_rows[threadIdx.x] = s_merged[threadIdx.x] = 0u;  // ordered by the first table's barriers
  const unsigned char* obs0 = e.obs;
  if constexpr (std::is_same<IN, ObsInline>::value) {
    obs0 = in.data;
    if (blockIdx.x == gridDim.x - 1)  // slot 0 keeps them for a later step without an upload
      for (int i = threadIdx.x * 8; i < in.bytes; i += kThreads * 8)
        *reinterpret_cast<unsigned long long*>(const_cast<unsigned char*>(e.obs) + i) =
            *reinterpret_cast<const unsigned long long*>(in.data + i);
  }
  int cb, ce;
  weighted_chunk<NCLK, WMODE>(e, t0, count, obs0, s_u64, s_cut, cb, ce);

  // ---------------------------------------------------------------- phase 1
  int cached = -1;
  int it = 0;
  for (int t = cb; t < ce; ++t, ++it) {

    const int f = __ldg(e.tile_filter + t);
    const FilterDesc* fd = e.desc + f;
    FilterCtrl* fc = e.ctrl + f;
    const unsigned epoch = fc->epoch;
    const bool lw_zero = fc->lw_zero != 0;
    const unsigned char* ob = obs0 + (size_t)(epoch % (unsigned)e.obs_slots) * e.obs_slot_bytes;
    const pf_filter_epoch_t* fe = reinterpret_cast<const pf_filter_epoch_t*>(ob) + f;
    const pf_sat_t* sats = reinterpret_cast<const pf_sat_t*>(ob + sizeof(pf_filter_epoch_t) * e.n_filters);
    const int eflags = fe->flags;
    int n_sat = fe->n_sat;
    if (n_sat > e.max_sats) {
      if (threadIdx.x == 0) raise_err(e, ERR_SAT_CAP);
      n_sat = e.max_sats;
    }
    if (n_sat < 0) n_sat = 0;
    const bool do_predict = (eflags & PF_EP_PREDICT) != 0;
    const bool do_weight = (eflags & PF_EP_WEIGHT) != 0;
    // the filter may resample this epoch: systematic builds its tiled integer CDF
    const bool may_rs = (do_weight || (eflags & PF_EP_RESAMPLE_CHECK)) && !(eflags & PF_EP_NO_RESAMPLE);
    const bool sys_q = RESAMPLER == PF_RESAMPLE_SYSTEMATIC && may_rs;
    if (t == fd->tile_begin && threadIdx.x == 0) {  // read after the barrier (phase 4, Megopolis)
      fc->sys_q_cur = sys_q ? 1 : 0;
      fc->eflags_cur = eflags;
      fc->epoch_cur = epoch;
      if (sys_q) fc->sys_u_cur = sys_offset_u(e, fd, epoch);
    }

    // the particles' loads are issued first: their memory latency overlaps the
    // satellite table of a new filter (FP64 geometry, two CTA barriers)
    const int n = fd->n;
    const int p0 = (t - fd->tile_begin) * kTile + (int)threadIdx.x * 4;
    const bool active = p0 < n;
    const long long base = fd->p_off;
    float* dst = fc->parity ? e.state0 : e.state1;
    float x[D][4];
    float lwv[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
    if (active) {
      load_particles<D>(e, fd, fc->parity ? e.state1 : e.state0, base, p0, n, fc->resample_flag != 0, x);
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d)
#pragma unroll
        for (int k = 0; k < 4; ++k) x[d][k] = 0.f;
    }
    if constexpr (WMODE == PF_WEIGHT_MIXTURE) {
      if (f != cached) {
        __shared__ MixSmem s_mix;
        build_mixture_table<NCLK>(e, fd, fc, fe, sats, n_sat, do_weight, t == fd->tile_begin, f, s_sat, s_grp, s_clk,
                                  s_mix);
        cached = f;
      }
    }
    if (WMODE != PF_WEIGHT_MIXTURE && f != cached) {  // satellite geometry of this filter (FP64 -> FP32 pairs)
      __syncthreads();   // nobody still reads the previous filter's table
      int my_c = 0;
      const pf_sat_t* sp = sats + fe->sat_offset + threadIdx.x;
      if (do_weight && threadIdx.x < n_sat) {
        my_c = sp->clk;
        my_c = my_c < 0 ? 0 : (my_c >= NCLK ? NCLK - 1 : my_c);
        s_clk[threadIdx.x] = (unsigned char)my_c;
      }
      __syncthreads();
      if (do_weight && threadIdx.x < n_sat) {
        const double* rot = fd->rot;
        double A[3];
        local_to_ecef(rot, fc->anchor, fc->shift[0], fc->shift[1], fc->shift[2], A);
        const int c = my_c;
        const double clkA = fc->clk_anchor[c] + (double)fc->shift[3 + c];
        double vx = sp->x - A[0], vy = sp->y - A[1], vz = sp->z - A[2];
        const double r0 = sqrt(vx * vx + vy * vy + vz * vz);
        const double inv = 1.0 / r0;
        vx *= inv; vy *= inv; vz *= inv;
        const float eE = (float)(rot[0] * vx + rot[1] * vy + rot[2] * vz);
        const float eN = (float)(rot[3] * vx + rot[4] * vy + rot[5] * vz);
        const float eU = (float)(rot[6] * vx + rot[7] * vy + rot[8] * vz);
        const float g = (float)inv;
        const float y = (float)(sp->pr - r0 - clkA);
        const float wq = WMODE == PF_WEIGHT_GAUSSIAN ? (float)((double)fd->wscale * sp->w) : (float)sp->w;
        int rank = 0;
        for (int s2 = 0; s2 < n_sat; ++s2) {
          const int c2 = s_clk[s2];
          rank += (c2 < c) || (c2 == c && s2 < (int)threadIdx.x);
        }
        if constexpr (WMODE == PF_WEIGHT_GENERIC)
          write_generic_entry(s_sat + kMixStride * rank, e, fd->sigma_pr, eE, eN, eU, g, y, (float)sp->w);
        else
          write_sat_entry(s_sat + kSatStride * rank, eE, eN, eU, g, y, wq);
      }
      if (threadIdx.x <= NCLK) {
        int cnt = 0;
        if (do_weight)
          for (int s2 = 0; s2 < n_sat; ++s2) cnt += s_clk[s2] < (int)threadIdx.x;
        s_grp[threadIdx.x] = cnt;
      }
      cached = f;
      __syncthreads();
    }

    if (active) {
      float lw0[4] = {0.f, 0.f, 0.f, 0.f};
      const bool need_prev = !lw_zero && (!do_weight || e.lw_mode == PF_LW_ACCUMULATE);
      if (need_prev) {
        const float4 v = __ldcs(reinterpret_cast<const float4*>(e.lw + base + p0));
        lw0[0] = v.x; lw0[1] = v.y; lw0[2] = v.z; lw0[3] = v.w;
      }
      float ds[D];
#pragma unroll
      for (int d = 0; d < D; ++d) ds[d] = -fc->shift[d];
      if (do_predict) {
        ds[0] += (float)fe->disp[0];
        ds[1] += (float)fe->disp[1];
        ds[2] += (float)fe->disp[2];
        predict4<D>(fd, p0, epoch, ds, x);
      } else {
#pragma unroll
        for (int d = 0; d < D; ++d)
#pragma unroll
          for (int k = 0; k < 4; ++k) x[d][k] += ds[d];
      }
#pragma unroll
      for (int d = 0; d < D; ++d)
        __stcs(reinterpret_cast<float4*>(dst + (size_t)d * e.p_total + base + p0),
               make_float4(x[d][0], x[d][1], x[d][2], x[d][3]));

      if (do_weight) {
        float2 lwp[2] = {f2(lw0[0], lw0[1]), f2(lw0[2], lw0[3])};
        float2 dx[2], dy[2], dz[2], nbb[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          dx[p] = f2(x[0][2 * p], x[0][2 * p + 1]);
          dy[p] = f2(x[1][2 * p], x[1][2 * p + 1]);
          dz[p] = f2(x[2][2 * p], x[2][2 * p + 1]);
          float2 bb = __fmul2_rn(dx[p], dx[p]);
          bb = __ffma2_rn(dy[p], dy[p], bb);
          bb = __ffma2_rn(dz[p], dz[p], bb);
          nbb[p] = f2(-bb.x, -bb.y);
        }
        if constexpr (WMODE == PF_WEIGHT_GENERIC) {
          float lim[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
          const float gate = e.lk_gate_m;
          if (gate > 0.f) {  // per-particle NLOS gate: drop |r| > gate unless too few satellites remain
            int kept[4] = {0, 0, 0, 0}, used = 0;
#pragma unroll
            for (int c = 0; c < NCLK; ++c) {
              const float2 ncb[2] = {f2(-x[3 + c][0], -x[3 + c][1]), f2(-x[3 + c][2], -x[3 + c][3])};
              generic_kept(s_sat, s_grp[c], s_grp[c + 1], dx, dy, dz, nbb, ncb, kept, used, gate);
            }
            const int need = used < 4 ? used : 4;
#pragma unroll
            for (int k = 0; k < 4; ++k) lim[k] = kept[k] >= need ? gate : INFINITY;
          }
          auto all_clocks = [&](auto type) {
#pragma unroll
            for (int c = 0; c < NCLK; ++c) {
              const float2 ncb[2] = {f2(-x[3 + c][0], -x[3 + c][1]), f2(-x[3 + c][2], -x[3 + c][3])};
              generic_pairs<decltype(type)::value>(s_sat, s_grp[c], s_grp[c + 1], dx, dy, dz, nbb, ncb, lwp, lim,
                                                   e.lk_huber_k, fd->inv_sigma_pr, -0.5f * (e.lk_nu + 1.f));
            }
          };
          if (e.lk_type == PF_LIK_STUDENT_T) all_clocks(LikType<PF_LIK_STUDENT_T>());
          else if (e.lk_type == PF_LIK_HUBER) all_clocks(LikType<PF_LIK_HUBER>());
          else if (e.lk_type == PF_LIK_GMM) all_clocks(LikType<PF_LIK_GMM>());
          else all_clocks(LikType<PF_LIK_GAUSSIAN>());
        }
#pragma unroll
        for (int c = 0; c < NCLK && WMODE != PF_WEIGHT_GENERIC; ++c) {
          const float2 ncb[2] = {f2(-x[3 + c][0], -x[3 + c][1]), f2(-x[3 + c][2], -x[3 + c][3])};
          const int s_end = s_grp[c + 1];
#pragma unroll 2
          for (int s = s_grp[c]; s < s_end; ++s) {
#pragma unroll
            for (int p = 0; p < 2; ++p) {
              if constexpr (WMODE == PF_WEIGHT_MIXTURE)
                sat_pair_mixture(s_sat + kMixStride * s, dx[p], dy[p], dz[p], nbb[p], ncb[p], lwp[p], fd);
              else
                sat_pair_update<WMODE>(s_sat + kSatStride * s, dx[p], dy[p], dz[p], nbb[p], ncb[p], lwp[p], fd);
            }
          }
        }
        lwv[0] = lwp[0].x; lwv[1] = lwp[0].y; lwv[2] = lwp[1].x; lwv[3] = lwp[1].y;
        __stcs(reinterpret_cast<float4*>(e.lw + base + p0), make_float4(lwv[0], lwv[1], lwv[2], lwv[3]));
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) lwv[k] = lw0[k];
        // reset weights live only in the control block: a resample test of
        // them (no weight pass) reads the array, so it is zeroed first
        if (lw_zero && (eflags & PF_EP_RESAMPLE_CHECK) && !(eflags & PF_EP_NO_RESAMPLE))
          __stcs(reinterpret_cast<float4*>(e.lw + base + p0), make_float4(0.f, 0.f, 0.f, 0.f));
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (p0 + k >= n) lwv[k] = -INFINITY;
    }

    // per-warp statistics, then one warp merges the warp rows into the tile row
    {
      float wm = fmaxf(fmaxf(lwv[0], lwv[1]), fmaxf(lwv[2], lwv[3]));
      wm = warp_max(wm);
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
      if (wm > -INFINITY) {
        const bool cov = (e.flags & PF_FLAG_COVARIANCE) != 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float w = exp2f((lwv[k] - wm) * 1.4426950408889634f);
          v[0] += w;
          v[1] = fmaf(w, w, v[1]);
#pragma unroll
          for (int d = 0; d < D; ++d) v[2 + d] = fmaf(w, x[d][k], v[2 + d]);
          if (cov) {
            const float wx = w * x[0][k], wy = w * x[1][k], wz = w * x[2][k];
            v[2 + D + 0] = fmaf(wx, x[0][k], v[2 + D + 0]);
            v[2 + D + 1] = fmaf(wx, x[1][k], v[2 + D + 1]);
            v[2 + D + 2] = fmaf(wx, x[2][k], v[2 + D + 2]);
            v[2 + D + 3] = fmaf(wy, x[1][k], v[2 + D + 3]);
            v[2 + D + 4] = fmaf(wy, x[2][k], v[2 + D + 4]);
            v[2 + D + 5] = fmaf(wz, x[2][k], v[2 + D + 5]);
          }
        }
      }
      const int idx = warp_transpose_sum16(v);
      // The warps' rows of tile `it` go to buffer it % kRowBufs and are merged
      // by warp it % 8, two tiles later: no warp waits for another unless it
      // runs kRowBufs tiles ahead, and every warp merges one tile in eight.
      // (One fixed merging warp, with two buffers and named barriers, kept the
      // eight warps in step and made that warp the tile's critical path: 256
      // Huber filters, 5.5M particles, 360.7 -> 352.5 us per step call; 64
      // learned filters of 100K, 433.9 -> 430.8 us; one filter of 1M particles,
      // 120.4 -> 119.2 us.)
      const int b = it % kRowBufs;
      if (it >= kRowBufs) cta_wait_reach(e, s_merged + b, (unsigned)(it / kRowBufs));  // the buffer is free
      // tiled integer CDF of the systematic resampler, segment level
      const double seg_sum = sys_q ? sys_segment_prefix(e, base, p0, active, lwv, wm, fd->K) : 0.0;
      if ((lane & 1) == 0 && idx < NV) s_wrow[b][warp][1 + idx] = v[0];
      if (lane == 0) {
        s_wrow[b][warp][0] = wm;
        s_wq[b][warp] = sys_q ? seg_sum : -1.0;  // -1: no CDF this step
      }
      __syncwarp();
      if (lane == 0) cta_red_release(s_rows + b);
      if (it >= kMergeLag && (it - kMergeLag) % kWarps == warp)
        merge_rows<NV, kWarps>(e, t - kMergeLag, it - kMergeLag, s_wrow, s_wq, s_rows, s_merged);
    }
  }
  for (int j = max(0, ce - cb - kMergeLag); j < ce - cb; ++j)  // the last tiles
    if (j % kWarps == warp) merge_rows<NV, kWarps>(e, cb + j, j, s_wrow, s_wq, s_rows, s_merged);
  grid_barrier(e, bar, gen);

  // ---------------------------------------------------------------- phase 2
  // Filter f_first + j is merged and decided by CTA j mod G.  With fewer
  // filters than CTAs the other CTAs start phase 4 (systematic) meanwhile.
  const int f_first = __ldg(e.tile_filter + t0), nf = __ldg(e.tile_filter + t0 + count - 1) - f_first + 1;
  for (int j = blockIdx.x; j < nf; j += gridDim.x) {
    const int f = f_first + j;
    const FilterDesc* fd = e.desc + f;
    FilterCtrl* fc = e.ctrl + f;
    const unsigned epoch = fc->epoch;
    const unsigned char* ob = obs0 + (size_t)(epoch % (unsigned)e.obs_slots) * e.obs_slot_bytes;
    const pf_filter_epoch_t* fe = reinterpret_cast<const pf_filter_epoch_t*>(ob) + f;
    const int eflags = fe->flags;
    MergedStats ms = merge_tiles<D>(e.part, fd->tile_begin, fd->n_tiles, s_maxtmp, s_dred);
    if (threadIdx.x == 0) {
      finalize_filter<D>(e, fd, fc, ms, epoch, fc->parity, fc->lw_zero != 0, eflags, (eflags & PF_EP_WEIGHT) != 0);
      s_dec_f = f;
      s_dec_rs = fc->resample_flag;
    }
    __syncthreads();
  }
  if constexpr (RESAMPLER == PF_RESAMPLE_SYSTEMATIC) {
    // Phase 4 needs only the first barrier: the tiled integer CDF is
    // complete once every tile is (speculative, as the owners decide at the
    // same time).  With few filters their owners sit it out (it overlaps
    // their merges); with many, every CTA takes a share after its merges.
    const int h0 = 4 * nf <= (int)gridDim.x ? nf : 0;  // first CTA of phase 4
    if ((int)blockIdx.x >= h0) {
      int b4, e4;
      chunk_of(t0, count, (int)blockIdx.x - h0, (int)gridDim.x - h0, b4, e4);
      epoch_sys_offspring(e, b4, e4, s_u64);
    }
    // no second barrier: the ancestors and segment markers are read first by
    // the next step, after this kernel has ended
  } else {
    // Megopolis: no second barrier either.  A CTA decides for the filter of
    // its tiles itself, with the owner's merge (the same function on the
    // same rows gives the same bits, hence the same decision) or, for the
    // filter it owns, with the owner's decision; epoch and flags come from
    // the snapshot phase 1 left (the owner advances the epoch meanwhile).
    int cf = -1;
    bool crs = false;
    cta_chunk(t0, count, cb, ce);  // here every tile costs the same
    for (int t = cb; t < ce; ++t) {
      const int f = __ldg(e.tile_filter + t);
      const FilterDesc* fd = e.desc + f;
      const FilterCtrl* fc = e.ctrl + f;
      if (f != cf) {  // CTA-uniform
        cf = f;
        if (f == s_dec_f) {
          crs = s_dec_rs != 0;
        } else {
          const MergedStats ms = merge_tiles<D>(e.part, fd->tile_begin, fd->n_tiles, s_maxtmp, s_dred);
          if (threadIdx.x == 0) s_dec_rs = resample_decision(e, fd, ms, ld_cg_int(&fc->eflags_cur)) ? 1 : 0;
          __syncthreads();
          crs = s_dec_rs != 0;
          __syncthreads();  // s_dec_rs is rewritten for the next filter
        }
      }
      if (crs) mego_tile(e, fd, ld_cg_u(&fc->epoch_cur), t);
    }
  }
}

}  // namespace pfb
