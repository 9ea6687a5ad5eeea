// pf_mlp.cu -- training and inference kernels of the per-satellite NLOS
// network (pf_mlp.cuh), on the tensor cores with BF16 operands and FP32
// accumulation.
//
// Loss per sample (label nlos in {0, 1}, bias b in metres):
//   L = BCE(sigmoid(o0), nlos) + nlos * ((mu - b) / 20 m)^2,  mu = 20 m softplus(o1)
// averaged over the batch.
//
// k_mlp_grad: each CTA takes rounds of 64 rows (4 warps x 16); per round a
// warp runs the forward pass and the backward pass of its rows on the tensor
// cores (dO -> dH2 = dO W3 masked by ReLU' -> dH1 = dH2 W2^T masked), stages
// activations and gradients in shared memory as BF16, and the CTA then forms
// the weight gradients dW = G^T H over the round's rows, again as MMAs (the bias
// gradients as products with ones), accumulated across rounds in registers.
// Per-CTA partial gradients go to a scratch array and k_mlp_reduce sums them in
// a fixed order (deterministic), then applies Adam or returns the gradient.
//
// A step on the default batch (8192 rows) is a latency chain: load, three
// layers forward, three back, weight gradients, reduction.  64 rows per CTA put
// it on 128 of 148 SMs (128 rows: on 64), transposed operands come by ldmatrix
// from padded rows (scalar two-byte loads before), and the two kernels of a step
// start while their predecessor drains.  Step of 8192 rows 32.8 -> 12.6 us, of
// 100,000 rows 239 -> 35 us.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>

#include "pf_mlp.cuh"
#include "pf_status.h"

namespace pfb {

constexpr int kMlpThreads = 128;
constexpr int kRows = 64;  // rows per CTA round
constexpr int kLdH = mlp_ld(kMlpH), kLdX = mlp_ld(kMlpIn);
constexpr int kMlpPart = kMlpParams + 1;  // floats per partial gradient (and its loss)

struct GradSmem {
  MlpSmem w;
  float x[kRows * kMlpIn];                     // inputs, FP32, cols 12..15 zero
  alignas(16) __nv_bfloat16 xb[kRows * kLdX];  // the same in BF16
  alignas(16) __nv_bfloat16 h1[kRows * kLdH];  // activations after ReLU
  alignas(16) __nv_bfloat16 h2[kRows * kLdH];
  alignas(16) __nv_bfloat16 g1[kRows * kLdH];  // dL/d(pre-activation) of layer 1
  alignas(16) __nv_bfloat16 g2[kRows * kLdH];  // of layer 2
  alignas(16) __nv_bfloat16 go[kRows * kLdX];  // dL/do (cols 0, 1), zero padded
  float loss[kMlpThreads / 32];
};

// The kernels of a step start while their predecessor, which writes what they
// read, still runs: their pointers are not __restrict__, so that no load may take
// the read-only path, whose lines are not kept in step with other SMs' stores, or
// move above the wait.
__device__ __forceinline__ void mlp_pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void mlp_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Store a BF16 A fragment (k-tile q) of rows [r0, r0+16) into a row-major
// [rows][64] BF16 array.
__device__ __forceinline__ void store_frag(__nv_bfloat16* dst, int r0, int q, int lane, const uint32_t (&a)[4]) {
  const int g = lane >> 2, t = lane & 3;
  *reinterpret_cast<uint32_t*>(dst + (r0 + g) * kLdH + 16 * q + 2 * t) = a[0];
  *reinterpret_cast<uint32_t*>(dst + (r0 + g + 8) * kLdH + 16 * q + 2 * t) = a[1];
  *reinterpret_cast<uint32_t*>(dst + (r0 + g) * kLdH + 16 * q + 8 + 2 * t) = a[2];
  *reinterpret_cast<uint32_t*>(dst + (r0 + g + 8) * kLdH + 16 * q + 8 + 2 * t) = a[3];
}

__device__ __forceinline__ float bf(uint32_t v, int hi) {
  return __bfloat162float(__ushort_as_bfloat16((unsigned short)(hi ? (v >> 16) : (v & 0xFFFFu))));
}

// Four 8x8 blocks of a row-major BF16 matrix, transposed: block j's rows start
// at the addresses of lanes 8j..8j+7.
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
}
// A fragment of the transposed operand: A[m][k] = src[k][m] for m in [16 mt,
// 16 mt + 16), k in [16 kt, 16 kt + 16); src is row-major with stride LD.
template <int LD>
__device__ __forceinline__ void a_frag_t(const __nv_bfloat16* src, int mt, int kt, int lane, uint32_t (&a)[4]) {
  const int j = lane >> 3, r = lane & 7;  // blocks: (k, m), (k, m + 8), (k + 8, m), (k + 8, m + 8)
  ldsm_x4_t(a, src + (16 * kt + (j >> 1) * 8 + r) * LD + 16 * mt + (j & 1) * 8);
}
// B fragments of n-tiles nt, nt + 1: B[k][n] = src[k][n], (b[0], b[1]) and (b[2], b[3]).
template <int LD>
__device__ __forceinline__ void b_frag_rows2(const __nv_bfloat16* src, int kt, int nt, int lane, uint32_t (&b)[4]) {
  const int j = lane >> 3, r = lane & 7;  // blocks: (k, n), (k + 8, n), (k, n + 8), (k + 8, n + 8)
  ldsm_x4_t(b, src + (16 * kt + (j & 1) * 8 + r) * LD + 8 * nt + (j >> 1) * 8);
}

__global__ void __launch_bounds__(kMlpThreads, 2)
    k_mlp_grad(const float* X, const float* Y, int n, const float* prm, float inv_n, float* partial) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GradSmem& S = *reinterpret_cast<GradSmem*>(smem_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  mlp_pdl_trigger();
  mlp_pdl_wait();
  mlp_stage(prm, S.w, kMlpThreads);

  // warp w: dW2t n-tiles 2w, 2w + 1 (all four m-tiles), dW1t m-tile w (both
  // n-tiles), dW3t n-tiles 2w, 2w + 1, bias gradients of m-tile w (db1, db2; warp 0 db3)
  float acc2[4][2][4], acc1[2][4], acc3[2][4], ab1[4], ab2[4], ab3[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    ab1[i] = ab2[i] = ab3[i] = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      acc1[h][i] = acc3[h][i] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) acc2[j][h][i] = 0.f;
    }
  }
  const uint32_t ones = 0x3F803F80u;  // two BF16 ones
  float lsum = 0.f;

  for (int base = blockIdx.x * kRows; base < n; base += gridDim.x * kRows) {
    __syncthreads();  // previous round's shared data consumed; weights staged
    for (int i = threadIdx.x; i < kRows * kMlpIn / 2; i += kMlpThreads) {
      const int r = i / (kMlpIn / 2), c = 2 * (i % (kMlpIn / 2));
      const bool in = base + r < n && c < kMlpFeat;
      const float x0 = in ? X[(size_t)(base + r) * kMlpFeat + c] : 0.f;
      const float x1 = in ? X[(size_t)(base + r) * kMlpFeat + c + 1] : 0.f;
      S.x[r * kMlpIn + c] = x0;
      S.x[r * kMlpIn + c + 1] = x1;
      *reinterpret_cast<uint32_t*>(S.xb + r * kLdX + c) = pack_bf16(x0, x1);
    }
    __syncthreads();
    const int r0 = warp * 16;
    MlpTile T;
    mlp_forward_tile(S.x + r0 * kMlpIn, S.w, lane, T);
    // loss and dL/do for rows r0 + g and r0 + g + 8 (lanes with t == 0)
    float d0[2] = {0.f, 0.f}, d1[2] = {0.f, 0.f};
    if (t == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = base + r0 + g + 8 * h;
        if (row < n) {
          const float o0 = T.o[2 * h], o1 = T.o[2 * h + 1];
          const float y = Y[2 * (size_t)row], b = Y[2 * (size_t)row + 1];
          const float p = sigmoidf_(o0);
          const float mu = kMuScale * softplusf(o1);
          const float e = (mu - b) / kMuScale;
          // BCE from the logit, stable for large |o0|
          const float bce = fmaxf(o0, 0.f) - o0 * y + log1pf(expf(-fabsf(o0)));
          lsum += bce + y * e * e;
          d0[h] = (p - y) * inv_n;
          d1[h] = y * 2.f * e * sigmoidf_(o1) * inv_n;  // d(e^2)/d(o1) = 2 e * softplus'(o1)
        }
      }
    }
    // dO as an A fragment (cols 0, 1 only) and into shared memory
    uint32_t ad[4];
    ad[0] = pack_bf16(d0[0], d1[0]);
    ad[1] = pack_bf16(d0[1], d1[1]);
    ad[2] = 0u;
    ad[3] = 0u;
    if (t != 0) ad[0] = ad[1] = 0u;
    {
      uint32_t* gr = reinterpret_cast<uint32_t*>(S.go + (r0 + g) * kLdX + 2 * t);
      uint32_t* gr8 = reinterpret_cast<uint32_t*>(S.go + (r0 + g + 8) * kLdX + 2 * t);
      gr[0] = ad[0];
      gr8[0] = ad[1];
      gr[4] = 0u;
      gr8[4] = 0u;
    }
    // dH2 = dO W3 (B[k = out][n = hidden] = W3t[out][hidden], zero for out >= 2), masked by ReLU'(H2)
    uint32_t gh2[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float c[2][4];
      uint32_t b[2];  // k 0..7 of n-tiles 2q, 2q + 1 (rows 2..7 are zero; k 8..15 likewise)
      {
        const __nv_bfloat16* p = S.w.w3t + (lane & 7) * kLdH + 16 * q + ((lane >> 3) & 1) * 8;
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
                     : "=r"(b[0]), "=r"(b[1])
                     : "r"((uint32_t)__cvta_generic_to_shared(p))
                     : "memory");
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < 4; ++i) c[h][i] = 0.f;
        mma_bf16(c[h], ad, b[h], 0u);
      }
      // mask: the same lane holds H2 at the same (row, col) in fragment q
      gh2[q][0] = pack_bf16(bf(T.h2[q][0], 0) > 0.f ? c[0][0] : 0.f, bf(T.h2[q][0], 1) > 0.f ? c[0][1] : 0.f);
      gh2[q][1] = pack_bf16(bf(T.h2[q][1], 0) > 0.f ? c[0][2] : 0.f, bf(T.h2[q][1], 1) > 0.f ? c[0][3] : 0.f);
      gh2[q][2] = pack_bf16(bf(T.h2[q][2], 0) > 0.f ? c[1][0] : 0.f, bf(T.h2[q][2], 1) > 0.f ? c[1][1] : 0.f);
      gh2[q][3] = pack_bf16(bf(T.h2[q][3], 0) > 0.f ? c[1][2] : 0.f, bf(T.h2[q][3], 1) > 0.f ? c[1][3] : 0.f);
    }
    // dH1 = dH2 W2^T (B[k = out2][n = in2] = W2t[out2][in2]), masked by ReLU'(H1)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float c[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) c[h][i] = 0.f;
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        uint32_t b[4];
        b_frag_rows2<kLdH>(S.w.w2t, kt, 2 * q, lane, b);
        mma_bf16(c[0], gh2[kt], b[0], b[1]);
        mma_bf16(c[1], gh2[kt], b[2], b[3]);
      }
      uint32_t gq[4];
      gq[0] = pack_bf16(bf(T.h1[q][0], 0) > 0.f ? c[0][0] : 0.f, bf(T.h1[q][0], 1) > 0.f ? c[0][1] : 0.f);
      gq[1] = pack_bf16(bf(T.h1[q][1], 0) > 0.f ? c[0][2] : 0.f, bf(T.h1[q][1], 1) > 0.f ? c[0][3] : 0.f);
      gq[2] = pack_bf16(bf(T.h1[q][2], 0) > 0.f ? c[1][0] : 0.f, bf(T.h1[q][2], 1) > 0.f ? c[1][1] : 0.f);
      gq[3] = pack_bf16(bf(T.h1[q][3], 0) > 0.f ? c[1][2] : 0.f, bf(T.h1[q][3], 1) > 0.f ? c[1][3] : 0.f);
      store_frag(S.g1, r0, q, lane, gq);
      store_frag(S.g2, r0, q, lane, gh2[q]);
      store_frag(S.h1, r0, q, lane, T.h1[q]);
      store_frag(S.h2, r0, q, lane, T.h2[q]);
    }
    __syncthreads();
    // weight gradients over the round: dW2t[out][in] = sum_s g2[s][out] h1[s][in]
#pragma unroll
    for (int kt = 0; kt < kRows / 16; ++kt) {
      uint32_t a[4], b[4];
      b_frag_rows2<kLdH>(S.h1, kt, 2 * warp, lane, b);
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        a_frag_t<kLdH>(S.g2, mt, kt, lane, a);
        mma_bf16(acc2[mt][0], a, b[0], b[1]);
        mma_bf16(acc2[mt][1], a, b[2], b[3]);
        if (mt == warp) mma_bf16(ab2, a, ones, ones);
      }
      // dW1t[out][in] = sum_s g1[s][out] x[s][in]
      a_frag_t<kLdH>(S.g1, warp, kt, lane, a);
      b_frag_rows2<kLdX>(S.xb, kt, 0, lane, b);
      mma_bf16(acc1[0], a, b[0], b[1]);
      mma_bf16(acc1[1], a, b[2], b[3]);
      mma_bf16(ab1, a, ones, ones);
      // dW3t[out][hid] = sum_s go[s][out] h2[s][hid]: rows out 0, 1 of the m-tile
      a_frag_t<kLdX>(S.go, 0, kt, lane, a);
      b_frag_rows2<kLdH>(S.h2, kt, 2 * warp, lane, b);
      mma_bf16(acc3[0], a, b[0], b[1]);
      mma_bf16(acc3[1], a, b[2], b[3]);
      if (warp == 0) mma_bf16(ab3, a, ones, ones);
    }
  }
  // per-CTA partial gradient
  float* P = partial + (size_t)blockIdx.x * kMlpPart;
  auto put2 = [&](int off, float v0, float v1) {  // the scratch is only known to be 4-byte aligned
    P[off] = v0;
    P[off + 1] = v1;
  };
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = 8 * (2 * warp + h) + 2 * t;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      put2(kOffW2 + (16 * mt + g) * kMlpH + i, acc2[mt][h][0], acc2[mt][h][1]);
      put2(kOffW2 + (16 * mt + g + 8) * kMlpH + i, acc2[mt][h][2], acc2[mt][h][3]);
    }
    put2(kOffW1 + (16 * warp + g) * kMlpIn + 8 * h + 2 * t, acc1[h][0], acc1[h][1]);
    put2(kOffW1 + (16 * warp + g + 8) * kMlpIn + 8 * h + 2 * t, acc1[h][2], acc1[h][3]);
    if (g < kMlpOut) put2(kOffW3 + g * kMlpH + i, acc3[h][0], acc3[h][1]);
  }
  if (t == 0) {  // the columns of a product with ones are equal
    P[kOffB1 + 16 * warp + g] = ab1[0];
    P[kOffB1 + 16 * warp + g + 8] = ab1[2];
    P[kOffB2 + 16 * warp + g] = ab2[0];
    P[kOffB2 + 16 * warp + g + 8] = ab2[2];
    if (warp == 0 && g < kMlpOut) P[kOffB3 + g] = ab3[0];
  }
  // loss sum (lanes with t == 0 hold row losses)
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if (lane == 0) S.loss[warp] = lsum;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < kMlpThreads / 32; ++w) s += S.loss[w];
    P[kMlpParams] = s;
  }
}

// Sum of the per-CTA partials in a fixed order (eight groups of CTAs, then the
// groups); then either the gradient (grad != nullptr) or one Adam step on prm
// (m, v moments, step >= 1).  32 parameters per CTA, one group per warp.
constexpr int kReduceGroups = 8;
__global__ void __launch_bounds__(32 * kReduceGroups)
    k_mlp_reduce(const float* partial, int nblk, float* grad, float* prm, float* m, float* v, int step,
                 float lr, float inv_n, float* loss) {
  __shared__ float s_sum[kReduceGroups][32];
  mlp_pdl_trigger();
  mlp_pdl_wait();
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (i <= kMlpParams) {
    const int per = (nblk + kReduceGroups - 1) / kReduceGroups, b0 = grp * per, b1 = min(nblk, b0 + per);
    const float* p = partial + (size_t)b0 * kMlpPart + i;
#pragma unroll 8
    for (int b = b0; b < b1; ++b, p += kMlpPart) s += __ldcg(p);
  }
  s_sum[grp][lane] = s;
  __syncthreads();
  if (grp != 0 || i > kMlpParams) return;
  s = 0.f;
#pragma unroll
  for (int q = 0; q < kReduceGroups; ++q) s += s_sum[q][lane];
  if (i == kMlpParams) {
    if (loss) *loss = s * inv_n;
    return;
  }
  if (grad) grad[i] = s;
  if (prm) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * m[i] + (1.f - b1) * s;
    const float vi = b2 * v[i] + (1.f - b2) * s * s;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.f - powf(b1, (float)step)), vh = vi / (1.f - powf(b2, (float)step));
    prm[i] -= lr * mh / (sqrtf(vh) + eps);
  }
}

// Inference: (p_nlos, mu) per row.  Bound by staging the weights and by the latency of
// three layers; with the rounds of 64 rows and the padded weight rows 8,192 rows
// 11.7 -> 7.3 us, 100,000 27.7 -> 13.7, 5M 838 -> 307 (rounds of 128 rows before).
__global__ void __launch_bounds__(kMlpThreads) k_mlp_forward(const float* __restrict__ X, int n,
                                                              const float* __restrict__ prm, float* __restrict__ out) {
  __shared__ MlpSmem W;
  __shared__ float xs[kRows * kMlpIn];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  mlp_stage(prm, W, kMlpThreads);
  for (int base = blockIdx.x * kRows; base < n; base += gridDim.x * kRows) {
    __syncthreads();
    for (int i = threadIdx.x; i < kRows * kMlpIn; i += kMlpThreads) {
      const int r = i / kMlpIn, c = i % kMlpIn;
      xs[i] = (base + r < n && c < kMlpFeat) ? X[(size_t)(base + r) * kMlpFeat + c] : 0.f;
    }
    __syncthreads();
    MlpTile T;
    mlp_forward_tile(xs + warp * 16 * kMlpIn, W, lane, T);
    if (t == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = base + warp * 16 + g + 8 * h;
        if (row < n) {
          out[2 * (size_t)row] = sigmoidf_(T.o[2 * h]);
          out[2 * (size_t)row + 1] = kMuScale * softplusf(T.o[2 * h + 1]);
        }
      }
    }
  }
}

// Two CTAs on each of 148 SMs.  A constant: the size of a caller's scratch follows
// from it, without a device at hand.
constexpr int kGradBlocks = 296;
constexpr int kMinPartials = 64;  // partial gradients that a caller's scratch must hold at least

// Launch that may start while the stream's previous kernel drains (the kernel
// waits for its results with griddepcontrol.wait).
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3((unsigned)grid);
  lc.blockDim = dim3((unsigned)block);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, kernel, args...);
}

}  // namespace pfb

using namespace pfb;

extern "C" {

int pf_mlp_param_count(void) { return kMlpParams; }

size_t pf_mlp_scratch_bytes(void) { return (size_t)kGradBlocks * kMlpPart * sizeof(float); }

// On as many CTAs as the rows fill, the SMs hold and the scratch has room for
// (gradient of 100,000 rows: 32 us with room for 296, 84 with 64).
static int grad_launch(const float* d_x, const float* d_y, int n, const float* d_params, float* d_scratch,
                       size_t scratch_bytes, int* nblk_out, cudaStream_t st) {
  const size_t room = scratch_bytes / (kMlpPart * sizeof(float));
  if (room < (size_t)kMinPartials) return set_err(PF_EINVAL, "scratch too small");
  const int nblk = (int)std::min({(size_t)kGradBlocks, ((size_t)n + kRows - 1) / kRows, room});
  const size_t smem = sizeof(GradSmem);
  cudaError_t e = cudaFuncSetAttribute((const void*)k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return set_err(PF_ECUDA, "mlp grad attribute: %s", cudaGetErrorString(e));
  e = launch_pdl(k_mlp_grad, nblk, kMlpThreads, smem, st, d_x, d_y, n, d_params, 1.0f / (float)n, d_scratch);
  if (e != cudaSuccess) return set_err(PF_ECUDA, "mlp grad launch: %s", cudaGetErrorString(e));
  *nblk_out = nblk;
  return PF_OK;
}

int pf_mlp_grad(const float* d_x, const float* d_y, int n, const float* d_params, float* d_grad, float* d_loss,
                void* d_scratch, size_t scratch_bytes, void* stream) {
  clear_err();
  if (!d_x || !d_y || !d_params || !d_grad || !d_scratch) return set_err(PF_EINVAL, "null pointer");
  if (n <= 0) return set_err(PF_EINVAL, "n must be > 0");
  cudaStream_t st = (cudaStream_t)stream;
  int nblk = 0, s;
  if ((s = grad_launch(d_x, d_y, n, d_params, (float*)d_scratch, scratch_bytes, &nblk, st)) != PF_OK) return s;
  cudaError_t e = launch_pdl(k_mlp_reduce, (kMlpParams + 32) / 32, 32 * kReduceGroups, 0, st, (const float*)d_scratch,
                             nblk, d_grad, (float*)nullptr, (float*)nullptr, (float*)nullptr, 0, 0.f,
                             1.0f / (float)n, d_loss);
  return e == cudaSuccess ? PF_OK : set_err(PF_ECUDA, "mlp reduce: %s", cudaGetErrorString(e));
}

int pf_mlp_adam_step(const float* d_x, const float* d_y, int n, float* d_params, float* d_m, float* d_v, int step,
                     float lr, float* d_loss, void* d_scratch, size_t scratch_bytes, void* stream) {
  clear_err();
  if (!d_x || !d_y || !d_params || !d_m || !d_v || !d_scratch) return set_err(PF_EINVAL, "null pointer");
  if (n <= 0 || step < 1 || !(lr > 0.f)) return set_err(PF_EINVAL, "bad n, step or lr");
  cudaStream_t st = (cudaStream_t)stream;
  int nblk = 0, s;
  if ((s = grad_launch(d_x, d_y, n, d_params, (float*)d_scratch, scratch_bytes, &nblk, st)) != PF_OK) return s;
  cudaError_t e = launch_pdl(k_mlp_reduce, (kMlpParams + 32) / 32, 32 * kReduceGroups, 0, st, (const float*)d_scratch,
                             nblk, (float*)nullptr, d_params, d_m, d_v, step, lr, 1.0f / (float)n, d_loss);
  return e == cudaSuccess ? PF_OK : set_err(PF_ECUDA, "mlp adam: %s", cudaGetErrorString(e));
}

int pf_mlp_forward(const float* d_x, int n, const float* d_params, float* d_out, void* stream) {
  clear_err();
  if (!d_x || !d_params || !d_out) return set_err(PF_EINVAL, "null pointer");
  if (n <= 0) return set_err(PF_EINVAL, "n must be > 0");
  const int nblk = std::min(1024, (n + kRows - 1) / kRows);
  k_mlp_forward<<<nblk, kMlpThreads, 0, (cudaStream_t)stream>>>(d_x, n, d_params, d_out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PF_OK : set_err(PF_ECUDA, "mlp forward: %s", cudaGetErrorString(e));
}

}  // extern "C"
