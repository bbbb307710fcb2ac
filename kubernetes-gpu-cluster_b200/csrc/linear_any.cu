// Shape-agnostic linear layer for layer-list models: any T / N / K and alignment, bfloat16 or float32 storage, fp32
// accumulation (float32 storage: in a fixed k order, so that a row's result does not depend on what else is in the launch; bfloat16: in the
// order of the kernel that the launch's sizes choose), optional row
// gather / scatter, per-row input scale, grouped rows (one weight slice per group: mixture-of-experts) or strided slices
// (block-diagonal projections), gated pairs (silu(x.w) * (x.w2)) and fp32 output or accumulation.  Tiles of 64 x 64
// outputs and 256 threads: float32 storage multiplies on the fp32 pipes (4 x 4 outputs per thread, operands staged in
// shared memory as fp32, true 32-bit products), bfloat16 storage on the tensor cores (mma.sync, further down).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "elt_access.cuh"
#include "hybrid_ops.h"

namespace kge {

__device__ __forceinline__ float act_apply(int act, float v) {
  switch (act) {
    case ACT_GELU_ERF: return 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
    case ACT_GELU_TANH: return 0.5f * v * (1.f + tanhf(0.79788456080286536f * (v + 0.044715f * v * v * v)));
    case ACT_SILU: return v / (1.f + expf(-v));
    case ACT_SIGMOID: return 1.f / (1.f + expf(-v));
    case ACT_TANH: return tanhf(v);
    case ACT_RELU2: { const float r = fmaxf(v, 0.f); return r * r; }
    case ACT_SOFTPLUS: return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v)));      // without overflow on either side
    default: return v;
  }
}
// softplus without overflow on either side, then the decay exp(-coef * softplus(v))
__device__ __forceinline__ float exp_decay(float coef, float v) { return expf(-coef * (fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))))); }

// the gated pair of two pre-activations (row scale applied)
__device__ __forceinline__ float glu_apply(const LinearArgs& a, float g, float u) {
  if (a.glu == GLU_CLAMPED_SIGMOID) {
    g = fminf(g, a.glu_limit);
    u = fminf(fmaxf(u, -a.glu_limit), a.glu_limit);
    return g / (1.f + expf(-a.glu_alpha * g)) * (u + 1.f);
  }
  return act_apply(ACT_SILU, g) * u;
}

constexpr int LBM = 64, LBN = 64, LBK = 16;

template <typename E, typename O, bool DUAL>
__global__ void __launch_bounds__(256) linear_any_kernel(LinearArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int z = blockIdx.z;
  int r0 = 0, r1 = a.T;
  if (a.group_off) { r0 = a.group_off[z]; r1 = a.group_off[z + 1]; }
  const int m0 = r0 + blockIdx.y * LBM;
  if (m0 >= r1) return;
  const int n0 = blockIdx.x * LBN;
  const E* x = (const E*)a.x + z * a.x_zs;
  const E* w = (const E*)a.w + z * a.w_zs;
  const E* w2 = DUAL ? (const E*)a.w2 + z * a.w_zs : nullptr;
  const E* bias = a.bias ? (const E*)a.bias + z * a.b_zs : nullptr;
  O* y = (O*)a.y + z * a.y_zs;
  __shared__ float xs[LBK][LBM + 1], ws[LBK][LBN + 1], ws2[DUAL ? LBK : 1][LBN + 1];
  __shared__ int xrow[LBM];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  if (tid < LBM) {
    const int r = m0 + tid;
    xrow[tid] = r < r1 ? (a.xrows ? a.xrows[r] : r) : -1;
  }
  __syncthreads();
  float acc[4][4] = {}, acc2[DUAL ? 4 : 1][4] = {};
  for (int k0 = 0; k0 < a.K; k0 += LBK) {
    for (int i = tid; i < LBM * LBK; i += 256) {
      const int r = i / LBK, k = i % LBK;
      const int xr = xrow[r];
      xs[k][r] = (xr >= 0 && k0 + k < a.K) ? ldf(x + (int64_t)xr * a.ldx + k0 + k) : 0.f;
      const int n = n0 + r;
      const bool ok = n < a.N && k0 + k < a.K;
      ws[k][r] = ok ? ldf(w + (int64_t)n * a.K + k0 + k) : 0.f;
      if (DUAL) ws2[k][r] = ok ? ldf(w2 + (int64_t)n * a.K + k0 + k) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < LBK; ++k) {
      float xv[4], wv[4], wv2[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { xv[i] = xs[k][ty * 4 + i]; wv[i] = ws[k][tx * 4 + i]; if (DUAL) wv2[i] = ws2[k][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
          if (DUAL) acc2[i][j] = fmaf(xv[i], wv2[j], acc2[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = m0 + ty * 4 + i;
    if (r >= r1) continue;
    const float s = a.row_scale ? a.row_scale[r] : 1.f;
    const int yr = a.yrows ? a.yrows[r] : r;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= a.N) continue;
      float v;
      if (DUAL) v = glu_apply(a, s * acc[i][j], s * acc2[i][j]);
      else {
        v = s * acc[i][j] + (bias ? ldf(bias + n) : 0.f);
        v = a.act == ACT_EXP_DECAY ? exp_decay(a.act_coef[n], v) : act_apply(a.act, v);
      }
      v *= a.alpha;
      O* dst = y + (int64_t)yr * a.ldy + n;
      if (a.accumulate) v += ldf(dst);
      stf(dst, v);
    }
  }
}

// bfloat16 operands: the same tiling on the tensor cores (mma.sync m16n8k16, fp32 accumulators).  Both operands are
// k-contiguous, which is exactly the row x col fragment layout, so the fragments are 32-bit loads from k-padded shared
// tiles.  Eight warps as 2 x 4, each 32 rows x 16 outputs; a row's sum is formed in the same k order whatever the launch holds.
constexpr int MPAD = 8;       // the k-tile is 32 wide for many rows and 64 for few (weight streaming: fewer, fatter round trips)

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// eight consecutive k of one row as one 16-byte register, zero beyond K or for a missing row; one 16-byte load when aligned
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* row, int k, int K, bool vec) {
  if (row && vec && k + 8 <= K) return *reinterpret_cast<const uint4*>(row + k);
  union { uint4 v; __nv_bfloat16 e[8]; } u;
#pragma unroll
  for (int i = 0; i < 8; ++i) u.e[i] = (row && k + i < K) ? row[k + i] : __float2bfloat16_rn(0.f);
  return u.v;
}

// one output from its sums (row scale applied): the gated pair, or bias and activation; then the multiplier
template <typename O>
__device__ __forceinline__ void linear_store(const LinearArgs& a, O* dst, const __nv_bfloat16* bias, int n, float s1, float s2) {
  float v;
  if (a.w2) v = glu_apply(a, s1, s2);
  else {
    v = s1 + (bias ? ldf(bias + n) : 0.f);
    v = a.act == ACT_EXP_DECAY ? exp_decay(a.act_coef[n], v) : act_apply(a.act, v);
  }
  v *= a.alpha;
  if (a.accumulate) v += ldf(dst);
  stf(dst, v);
}

template <typename O, bool DUAL, int MBK>
__global__ void __launch_bounds__(256) linear_mma_kernel(LinearArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  typedef __nv_bfloat16 E;
  const int z = blockIdx.z;
  int r0 = 0, r1 = a.T;
  if (a.group_off) { r0 = a.group_off[z]; r1 = a.group_off[z + 1]; }
  const int m0 = r0 + blockIdx.y * LBM;
  if (m0 >= r1) return;
  const int n0 = blockIdx.x * LBN;
  const E* x = (const E*)a.x + z * a.x_zs;
  const E* w = (const E*)a.w + z * a.w_zs;
  const E* w2 = DUAL ? (const E*)a.w2 + z * a.w_zs : nullptr;
  const E* bias = a.bias ? (const E*)a.bias + z * a.b_zs : nullptr;
  O* y = (O*)a.y + z * a.y_zs;
  __shared__ __align__(16) E xs[LBM][MBK + MPAD], ws[LBN][MBK + MPAD], ws2[DUAL ? LBN : 1][MBK + MPAD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
  // staging: thread -> (row tid / 4, eight k at (tid % 4) * 8)
  const int sr = tid >> 2, sk = (tid & 3) * 8;
  const int gr = m0 + sr;
  const E* xrow = gr < r1 ? x + (int64_t)(a.xrows ? a.xrows[gr] : gr) * a.ldx : nullptr;
  const E* wrow = n0 + sr < a.N ? w + (int64_t)(n0 + sr) * a.K : nullptr;
  const E* w2row = (DUAL && n0 + sr < a.N) ? w2 + (int64_t)(n0 + sr) * a.K : nullptr;
  const bool xvec = ((reinterpret_cast<uintptr_t>(x) & 15) == 0) && a.ldx % 8 == 0;
  const bool wvec = ((reinterpret_cast<uintptr_t>(w) & 15) == 0) && a.K % 8 == 0 && (!DUAL || (reinterpret_cast<uintptr_t>(w2) & 15) == 0);
  float acc[2][2][4] = {}, acc2[DUAL ? 2 : 1][2][4] = {};
  // the next k-tile travels from global memory to registers while the tensor cores work on the current one
  constexpr int NU = MBK / 32;                 // 16-byte pieces per thread, operand and k-tile
  uint4 px[NU], pw[NU], pw2[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    px[u] = load8(xrow, sk + u * 32, a.K, xvec);
    pw[u] = load8(wrow, sk + u * 32, a.K, wvec);
    pw2[u] = DUAL ? load8(w2row, sk + u * 32, a.K, wvec) : make_uint4(0u, 0u, 0u, 0u);
  }
  for (int k0 = 0; k0 < a.K; k0 += MBK) {
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      *reinterpret_cast<uint4*>(&xs[sr][sk + u * 32]) = px[u];
      *reinterpret_cast<uint4*>(&ws[sr][sk + u * 32]) = pw[u];
      if (DUAL) *reinterpret_cast<uint4*>(&ws2[sr][sk + u * 32]) = pw2[u];
    }
    __syncthreads();
    if (k0 + MBK < a.K) {
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        px[u] = load8(xrow, k0 + MBK + sk + u * 32, a.K, xvec);
        pw[u] = load8(wrow, k0 + MBK + sk + u * 32, a.K, wvec);
        if (DUAL) pw2[u] = load8(w2row, k0 + MBK + sk + u * 32, a.K, wvec);
      }
    }
#pragma unroll
    for (int ks = 0; ks < MBK / 16; ++ks) {
      const int kc = ks * 16 + (lane & 3) * 2;
      uint32_t af[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm + i * 16 + (lane >> 2);
        af[i][0] = *reinterpret_cast<const uint32_t*>(&xs[r][kc]);
        af[i][1] = *reinterpret_cast<const uint32_t*>(&xs[r + 8][kc]);
        af[i][2] = *reinterpret_cast<const uint32_t*>(&xs[r][kc + 8]);
        af[i][3] = *reinterpret_cast<const uint32_t*>(&xs[r + 8][kc + 8]);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int n = wn + j * 8 + (lane >> 2);
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(&ws[n][kc]), b1 = *reinterpret_cast<const uint32_t*>(&ws[n][kc + 8]);
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_bf16_16816(acc[i][j], af[i], b0, b1);
        if (DUAL) {
          const uint32_t c0 = *reinterpret_cast<const uint32_t*>(&ws2[n][kc]), c1 = *reinterpret_cast<const uint32_t*>(&ws2[n][kc + 8]);
#pragma unroll
          for (int i = 0; i < 2; ++i) mma_bf16_16816(acc2[i][j], af[i], c0, c1);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int r = m0 + wm + i * 16 + (lane >> 2) + hh * 8;
      if (r >= r1) continue;
      const float sc = a.row_scale ? a.row_scale[r] : 1.f;
      const int yr = a.yrows ? a.yrows[r] : r;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int n = n0 + wn + j * 8 + (lane & 3) * 2 + c;
          if (n >= a.N) continue;
          const float s1 = acc[i][j][hh * 2 + c];
          float v;
          if (DUAL) v = glu_apply(a, sc * s1, sc * acc2[i][j][hh * 2 + c]);
          else {
            v = sc * s1 + (bias ? ldf(bias + n) : 0.f);
            v = a.act == ACT_EXP_DECAY ? exp_decay(a.act_coef[n], v) : act_apply(a.act, v);
          }
          v *= a.alpha;
          O* dst = y + (int64_t)yr * a.ldy + n;
          if (a.accumulate) v += ldf(dst);
          stf(dst, v);
        }
    }
}

// Few rows, 16-byte aligned operands, long sums: the weights are the traffic, so they stream through a ring of four k-tiles filled by
// cp.async three ahead; tiles of 64 rows x 64 weight rows (gated pairs: 32 of each matrix), the same fragments and the same
// order of summation as above.  Row tiles of 16 without rows (experts with few tokens) are not multiplied.
constexpr int SBK = 64, SST = 4, SLD = SBK + MPAD;
constexpr size_t LINEAR_STREAM_SMEM = (size_t)SST * (LBM + LBN) * SLD * 2;

template <typename O, bool DUAL>
__global__ void __launch_bounds__(256) linear_stream_kernel(LinearArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  typedef __nv_bfloat16 E;
  constexpr int BN = DUAL ? LBN / 2 : LBN, NT = BN / 32;      // outputs per tile; 8-output tiles per warp
  const int z = blockIdx.z;
  int r0 = 0, r1 = a.T;
  if (a.group_off) { r0 = a.group_off[z]; r1 = a.group_off[z + 1]; }
  const int m0 = r0 + blockIdx.y * LBM;
  if (m0 >= r1) return;
  const int n0 = blockIdx.x * BN, mrows = r1 - m0;
  const E* x = (const E*)a.x + z * a.x_zs;
  const E* w = (const E*)a.w + z * a.w_zs;
  const E* w2 = DUAL ? (const E*)a.w2 + z * a.w_zs : nullptr;
  const E* bias = a.bias ? (const E*)a.bias + z * a.b_zs : nullptr;
  O* y = (O*)a.y + z * a.y_zs;
  extern __shared__ __align__(16) unsigned char ls_raw[];
  E* xs = reinterpret_cast<E*>(ls_raw);                       // [SST][LBM][SLD]
  E* ws = xs + SST * LBM * SLD;                               // [SST][LBN][SLD]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 2) * 32, wn = (warp & 3) * (NT * 8);
  // staging: thread -> rows tid / 8 and tid / 8 + 32 of both tiles, eight k at (tid % 8) * 8
  const int sr = tid >> 3, sk = (tid & 7) * 8;
  const E *xp[2], *wp[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int gr = m0 + sr + 32 * u;
    xp[u] = gr < r1 ? x + (int64_t)(a.xrows ? a.xrows[gr] : gr) * a.ldx : nullptr;
    const int n = n0 + (DUAL ? sr : sr + 32 * u);
    wp[u] = n < a.N ? (DUAL && u ? w2 : w) + (int64_t)n * a.K : nullptr;
  }
  auto cp = [&](E* dst, const E* row, int k) {
    const bool ok = row != nullptr && k < a.K;
    const int sz = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(ok ? row + k : w), "r"(sz));
  };
  const int nk = (a.K + SBK - 1) / SBK;
  auto stage = [&](int kt) {
    if (kt < nk) {
      const int st = kt % SST, k = kt * SBK + sk;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (sr + 32 * u < ((mrows + 15) & ~15)) cp(xs + (st * LBM + sr + 32 * u) * SLD + sk, xp[u], k);
        cp(ws + (st * LBN + sr + 32 * u) * SLD + sk, wp[u], k);
      }
    }
    asm volatile("cp.async.commit_group;");
  };
#pragma unroll
  for (int i = 0; i < SST - 1; ++i) stage(i);
  float acc[2][NT][4] = {}, acc2[DUAL ? 2 : 1][NT][4] = {};
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(SST - 2) : "memory");
    __syncthreads();                                          // this k-tile has landed; the readers of the one refilled next are done
    stage(kt + SST - 1);
    const E* xt = xs + kt % SST * LBM * SLD;
    const E* wt = ws + kt % SST * LBN * SLD;
#pragma unroll
    for (int ks = 0; ks < SBK / 16; ++ks) {
      const int kc = ks * 16 + (lane & 3) * 2;
      uint32_t b[NT][2], c[DUAL ? NT : 1][2];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const E* p = wt + (wn + j * 8 + (lane >> 2)) * SLD + kc;
        b[j][0] = *reinterpret_cast<const uint32_t*>(p); b[j][1] = *reinterpret_cast<const uint32_t*>(p + 8);
        if (DUAL) { c[j][0] = *reinterpret_cast<const uint32_t*>(p + 32 * SLD); c[j][1] = *reinterpret_cast<const uint32_t*>(p + 32 * SLD + 8); }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (wm + i * 16 < mrows) {
          const E* p = xt + (wm + i * 16 + (lane >> 2)) * SLD + kc;
          const uint32_t af[4] = {*reinterpret_cast<const uint32_t*>(p), *reinterpret_cast<const uint32_t*>(p + 8 * SLD), *reinterpret_cast<const uint32_t*>(p + 8),
                                  *reinterpret_cast<const uint32_t*>(p + 8 * SLD + 8)};
#pragma unroll
          for (int j = 0; j < NT; ++j) {
            mma_bf16_16816(acc[i][j], af, b[j][0], b[j][1]);
            if (DUAL) mma_bf16_16816(acc2[i][j], af, c[j][0], c[j][1]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int r = m0 + wm + i * 16 + (lane >> 2) + hh * 8;
      if (r >= r1) continue;
      const float sc = a.row_scale ? a.row_scale[r] : 1.f;
      const int yr = a.yrows ? a.yrows[r] : r;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int n = n0 + wn + j * 8 + (lane & 3) * 2 + q;
          if (n < a.N) linear_store(a, y + (int64_t)yr * a.ldy + n, bias, n, sc * acc[i][j][hh * 2 + q], DUAL ? sc * acc2[DUAL ? i : 0][j][hh * 2 + q] : 0.f);
        }
    }
}

// Many rows, a short sum, fp32 output (the second half of a low-rank pair): the output is the traffic.  128 x 128 tiles whose operands
// are staged whole (K <= 256) with cp.async; eight warps of 64 rows x 32 outputs, fragments by ldmatrix, the same order of summation
// as above, two outputs per store.  Strided slices (block-diagonal gates) are the grid's third dimension: 2312 rows by 16 blocks of 160 x 160
// 38 us in the 64-row tiles of linear_mma_kernel, 23 here.
constexpr int WBM = 128, WBN = 128, WMAXK = 256;

__device__ __forceinline__ void la_ldsm4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

template <int ACT>
__global__ void __launch_bounds__(256) linear_short_kernel(LinearArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  typedef __nv_bfloat16 E;
  extern __shared__ __align__(16) unsigned char lw_raw[];
  const int pitch = a.K + MPAD, pieces = a.K / 8;
  E* xs = reinterpret_cast<E*>(lw_raw);                       // [WBM][pitch]
  E* ws = xs + WBM * pitch;                                   // [WBN][pitch]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, m0 = blockIdx.y * WBM, n0 = blockIdx.x * WBN, z = blockIdx.z;
  const E *x = (const E*)a.x + z * a.x_zs, *w = (const E*)a.w + z * a.w_zs, *b = a.bias ? (const E*)a.bias + z * a.b_zs : nullptr;
  for (int i = tid; i < (WBM + WBN) * pieces; i += 256) {
    const int r = i / pieces, k = i % pieces * 8;
    const bool isx = r < WBM;
    const int g = isx ? m0 + r : n0 + r - WBM;
    const bool ok = isx ? g < a.T : g < a.N;
    const E* src = isx ? x + (ok ? (int64_t)g * a.ldx + k : 0) : w + (ok ? (int64_t)g * a.K + k : 0);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(xs + r * pitch + k)), "l"(src), "r"(ok ? 16 : 0));
  }
  asm volatile("cp.async.commit_group;");
  const int wm = (warp >> 2) * 64, wn = (warp & 3) * 32, lr = lane & 7, lm = lane >> 3;
  float2 bias[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + wn + j * 8 + (lane & 3) * 2;
    bias[j] = make_float2(b && n < a.N ? ldf(b + n) : 0.f, b && n + 1 < a.N ? ldf(b + n + 1) : 0.f);
  }
  float acc[4][4][4] = {};
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (n0 + wn >= a.N) return;                                 // no outputs, and no barrier behind
  for (int k = 0; k < a.K; k += 16) {
    uint32_t bf[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) la_ldsm4(bf[j], ws + (wn + j * 16 + (lm >> 1) * 8 + lr) * pitch + k + (lm & 1) * 8);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t af[4];
      la_ldsm4(af, xs + (wm + i * 16 + (lm & 1) * 8 + lr) * pitch + k + (lm >> 1) * 8);
#pragma unroll
      for (int j = 0; j < 4; ++j) mma_bf16_16816(acc[i][j], af, bf[j >> 1][(j & 1) * 2], bf[j >> 1][(j & 1) * 2 + 1]);
    }
  }
  float* y = (float*)a.y + z * a.y_zs;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int r = m0 + wm + i * 16 + (lane >> 2) + hh * 8;
      if (r >= a.T) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + wn + j * 8 + (lane & 3) * 2;
        if (n >= a.N) continue;                               // N is even: a pair is inside or outside
        float u = acc[i][j][hh * 2] + bias[j].x, v = acc[i][j][hh * 2 + 1] + bias[j].y;
        if (ACT == ACT_EXP_DECAY) { u = exp_decay(a.act_coef[n], u); v = exp_decay(a.act_coef[n + 1], v); }
        else { u = act_apply(ACT, u); v = act_apply(ACT, v); }
        *reinterpret_cast<float2*>(y + (int64_t)r * a.ldy + n) = make_float2(u * a.alpha, v * a.alpha);
      }
    }
}

// Few outputs (gates, routers: up to 32 columns), fp32: the rows of x are the traffic.  A CTA takes 16 rows; its eight warps
// interleave over K in chunks of 64 and add their sums in warp order in shared memory.  mma.m16n8k16 with the rows as M: the order
// of a contraction is free, so lane t of a quad takes 16 consecutive bytes of each 32-number piece of both operands, copied by
// cp.async into slots that only it reads (no barrier in the loop).  2312 x 2048 by 8: 5.6 us, 2 rows: 4.8 us (64-row tiles of
// the kernels above: 47 and 17).
template <int NT>
__global__ void __launch_bounds__(256) linear_narrow_kernel(LinearArgs a) {
  constexpr int S = 3, PIECES = 2 * (NT + 2);
  typedef __nv_bfloat16 E;
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint4 ln_ring[];             // [warp][stage][piece][lane]
  __shared__ float part[8][16][NT * 8 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, m0 = blockIdx.x * 16;
  const int chunks = (a.K + 63) / 64, mine = chunks > warp ? (chunks - warp + 7) / 8 : 0;
  const E* wrow[NT];
  const E* xrow[2];
#pragma unroll
  for (int j = 0; j < NT; ++j) wrow[j] = (const E*)a.w + (int64_t)min(j * 8 + g, a.N - 1) * a.K + t * 8;
#pragma unroll
  for (int i = 0; i < 2; ++i) xrow[i] = (const E*)a.x + (int64_t)min(m0 + g + 8 * i, a.T - 1) * a.ldx + t * 8;
  uint4* slot0 = ln_ring + (warp * S * PIECES) * 32 + lane;
  auto copy = [&](uint4* dst, const E* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(in ? src : (const E*)a.w), "r"(in ? 16u : 0u) : "memory");
  };
  auto stage = [&](int i) {
    if (i < mine) {
      uint4* dst = slot0 + (i % S) * PIECES * 32;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = (warp + i * 8) * 64 + h * 32;
        const bool in = k + t * 8 < a.K;
#pragma unroll
        for (int j = 0; j < NT; ++j) copy(dst + (2 * j + h) * 32, wrow[j] + k, in && j * 8 + g < a.N);      // no reads of one row in the place of many
#pragma unroll
        for (int j = 0; j < 2; ++j) copy(dst + (2 * (NT + j) + h) * 32, xrow[j] + k, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pdl_wait();
  float acc[NT][4] = {};
#pragma unroll
  for (int i = 0; i < S - 1; ++i) stage(i);
#pragma unroll 1
  for (int i = 0; i < mine; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    const uint4* src = slot0 + (i % S) * PIECES * 32;
    uint4 wv[NT][2], xv[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int j = 0; j < NT; ++j) wv[j][h] = src[(2 * j + h) * 32];
#pragma unroll
      for (int j = 0; j < 2; ++j) xv[j][h] = src[(2 * (NT + j) + h) * 32];
    }
    stage(i + S - 1);                                          // into the stage that the previous turn read
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t a0[4] = {xv[0][h].x, xv[1][h].x, xv[0][h].y, xv[1][h].y}, a1[4] = {xv[0][h].z, xv[1][h].z, xv[0][h].w, xv[1][h].w};
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        mma_bf16_16816(acc[j], a0, wv[j][h].x, wv[j][h].y);
        mma_bf16_16816(acc[j], a1, wv[j][h].z, wv[j][h].w);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) part[warp][g + 8 * (q >> 1)][j * 8 + t * 2 + (q & 1)] = acc[j][q];
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * a.N; i += 256) {
    const int r = i / a.N, n = i % a.N;
    if (m0 + r >= a.T) break;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += part[w][r][n];
    linear_store(a, (float*)a.y + (int64_t)(m0 + r) * a.ldy + n, (const E*)a.bias, n, v, 0.f);
  }
}
// The general kernels keep short sums over many rows where three or four column tiles are in use: a CTA would set up 144 KB of ring
// for six chunks of K (us here and there by 32 columns: 16384 x 256 13.9 and 8.3, 16384 x 264 16.6 and 13.9, 8192 x 264 10.0 and 9.4;
// but 16384 x 384 14.5 and 16.2, 4096 x 264 5.9 and 8.1).
static bool linear_narrow_ok(const LinearArgs& a) {
  if (a.N > 16 && a.K < 384 && a.T > 4096) return false;
  return a.elt == KGE_ELT_BF16 && a.out_f32 && !a.w2 && !a.group_off && !a.xrows && !a.yrows && !a.row_scale && a.nz == 1 && a.N <= 32 && a.K >= 256 && a.K % 8 == 0 && a.ldx % 8 == 0 &&
         ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w)) & 15) == 0;
}
template <int NT>
static int launch_linear_narrow(const LinearArgs& a, cudaStream_t st) {
  constexpr int smem = 8 * 3 * 2 * (NT + 2) * 512;
  KGE_CUDA_OK(cudaFuncSetAttribute(linear_narrow_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  KGE_CUDA_OK(launch_pdl(linear_narrow_kernel<NT>, dim3((a.T + 15) / 16), dim3(256), smem, st, a));
  return 0;
}

// A few rows (up to 8 in all slices together): every weight is used once or twice, so a warp streams its own weight rows as in gemm_rows.cuh:
// mma.m16n8k16 with the rows as M, a lane copies 16 consecutive bytes of each 32-number piece of the weights by cp.async into slots that only
// it reads, the eight warps of a CTA interleave over K in chunks of 64 and add their sums in warp order.  A CTA has 8 outputs (gated pairs:
// 8 of either matrix) of one slice; of groups only as many as there are rows are launched.  Strided slices ask for their first weights before the wait; which
// groups have rows is the previous kernel's result.  us on cold weights in the ring of linear_stream_kernel or the tiles of
// linear_mma_kernel and here: 4 rows in 4 of 16 experts, gated 2 x 1024 x 2048 25.8 / 11.4, 2048 x 1024 15.5 / 9.6, 2 rows by 16 blocks of
// 160 x 160 7.8 / 4.4.
constexpr int FEW_ROWS = 8, FEW_S = 4;
template <typename O, bool DUAL>
__global__ void __launch_bounds__(256) linear_few_kernel(LinearArgs a) {
  constexpr int NW = DUAL ? 2 : 1, PIECES = 2 * (NW + 1);
  typedef __nv_bfloat16 E;
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint4 lf_ring[];             // [warp][stage][piece][lane]
  __shared__ float part[8][FEW_ROWS][NW * 8 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, n0 = blockIdx.x * 8;
  const int chunks = (a.K + 63) / 64, mine = chunks > warp ? (chunks - warp + 7) / 8 : 0;
  int z = a.group_off ? 0 : blockIdx.y;
  const E* wrow[NW];
  auto rows_of = [&] {
#pragma unroll
    for (int j = 0; j < NW; ++j) wrow[j] = (const E*)(j ? a.w2 : a.w) + z * a.w_zs + (int64_t)min(n0 + g, a.N - 1) * a.K + t * 8;
  };
  rows_of();
  uint4* slot0 = lf_ring + (warp * FEW_S * PIECES) * 32 + lane;
  auto copy = [&](uint4* dst, const E* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(in ? src : (const E*)a.w), "r"(in ? 16u : 0u) : "memory");
  };
  auto copy_w = [&](int i) {
    uint4* dst = slot0 + (i % FEW_S) * PIECES * 32;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = (warp + i * 8) * 64 + h * 32;
#pragma unroll
      for (int j = 0; j < NW; ++j) copy(dst + (2 * j + h) * 32, wrow[j] + k, k + t * 8 < a.K && n0 + g < a.N);
    }
  };
  if (!a.group_off) {
#pragma unroll
    for (int i = 0; i < FEW_S - 1; ++i)
      if (i < mine) copy_w(i);
  }
  pdl_wait();
  int r0 = 0, rows = a.T;
  if (a.group_off) {
    // group number blockIdx.y of those that have rows
    int left = blockIdx.y, found = -1;
    for (int z0 = 0; z0 < a.nz && found < 0; z0 += 32) {
      const int i = z0 + lane, lo = i < a.nz ? a.group_off[i] : 0, hi = i < a.nz ? a.group_off[i + 1] : 0;
      uint32_t some = __ballot_sync(0xffffffffu, hi > lo);
      if (left < __popc(some)) {
        for (; left > 0; --left) some &= some - 1;
        found = __ffs(some) - 1;
        z = z0 + found;
        r0 = __shfl_sync(0xffffffffu, lo, found);
        rows = __shfl_sync(0xffffffffu, hi, found) - r0;
      }
      left -= __popc(some);
    }
    if (found < 0) return;                                     // (no copy is under way)
    rows_of();
  }
  const int r = r0 + min(g, rows - 1);
  const E* xrow = (const E*)a.x + z * a.x_zs + (int64_t)(a.xrows ? a.xrows[r] : r) * a.ldx + t * 8;
  auto copy_x = [&](int i) {
    uint4* dst = slot0 + ((i % FEW_S) * PIECES + 2 * NW) * 32;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = (warp + i * 8) * 64 + h * 32;
      copy(dst + h * 32, xrow + k, k + t * 8 < a.K && g < rows);
    }
  };
#pragma unroll
  for (int i = 0; i < FEW_S - 1; ++i) {
    if (i < mine) {
      if (a.group_off) copy_w(i);
      copy_x(i);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[NW][4] = {};
#pragma unroll 1
  for (int i = 0; i < mine; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FEW_S - 2) : "memory");
    const uint4* src = slot0 + (i % FEW_S) * PIECES * 32;
    uint4 wv[NW][2], xv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int j = 0; j < NW; ++j) wv[j][h] = src[(2 * j + h) * 32];
      xv[h] = src[(2 * NW + h) * 32];
    }
    if (i + FEW_S - 1 < mine) { copy_w(i + FEW_S - 1); copy_x(i + FEW_S - 1); }      // into the stage that the previous turn read
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t a0[4] = {xv[h].x, 0u, xv[h].y, 0u}, a1[4] = {xv[h].z, 0u, xv[h].w, 0u};
#pragma unroll
      for (int j = 0; j < NW; ++j) {
        mma_bf16_16816(acc[j], a0, wv[j][h].x, wv[j][h].y);
        mma_bf16_16816(acc[j], a1, wv[j][h].z, wv[j][h].w);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NW; ++j)
#pragma unroll
    for (int q = 0; q < 2; ++q) part[warp][g][j * 8 + t * 2 + q] = acc[j][q];
  __syncthreads();
  const int row = threadIdx.x >> 3, col = threadIdx.x & 7, n = n0 + col;
  if (row < rows && n < a.N) {
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      s1 += part[w][row][col];
      if (DUAL) s2 += part[w][row][8 + col];
    }
    const float sc = a.row_scale ? a.row_scale[r0 + row] : 1.f;
    const int yr = a.yrows ? a.yrows[r0 + row] : r0 + row;
    linear_store(a, (O*)a.y + z * a.y_zs + (int64_t)yr * a.ldy + n, a.bias ? (const E*)a.bias + z * a.b_zs : nullptr, n, sc * s1, sc * s2);
  }
}
static bool linear_few_ok(const LinearArgs& a) {
  return a.elt == KGE_ELT_BF16 && a.T <= FEW_ROWS && a.K % 8 == 0 && a.K >= 64 && a.N <= 32768 && a.ldx % 8 == 0 && a.x_zs % 8 == 0 && a.w_zs % 8 == 0 && a.nz <= 65535 &&
         ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.w2)) & 15) == 0;
}
static int launch_linear_few(const LinearArgs& a, cudaStream_t st) {
  auto kern = a.out_f32 ? (a.w2 ? linear_few_kernel<float, true> : linear_few_kernel<float, false>)
                        : (a.w2 ? linear_few_kernel<__nv_bfloat16, true> : linear_few_kernel<__nv_bfloat16, false>);
  const int smem = 8 * FEW_S * 2 * (a.w2 ? 3 : 2) * 512;
  KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  KGE_CUDA_OK(launch_pdl(kern, dim3((a.N + 7) / 8, a.group_off ? std::min(a.nz, a.T) : a.nz), dim3(256), smem, st, a));
  return 0;
}

static bool linear_short_ok(const LinearArgs& a) {
  return a.elt == KGE_ELT_BF16 && a.out_f32 && !a.w2 && !a.group_off && !a.xrows && !a.yrows && !a.row_scale && !a.accumulate && a.nz <= 65535 && (a.nz == 1 || (a.act == ACT_NONE && a.x_zs % 8 == 0 && a.w_zs % 8 == 0 && a.y_zs % 2 == 0)) && a.T > 256 && a.K % 16 == 0 && a.K <= WMAXK &&
         a.N % 2 == 0 && a.ldy % 2 == 0 && a.ldx % 8 == 0 && (a.T + WBM - 1) / WBM <= 65535 && (a.act == ACT_NONE || a.act == ACT_SOFTPLUS || a.act == ACT_EXP_DECAY) &&
         ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w)) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.y) & 7) == 0;
}

int linear_any(const LinearArgs& a, cudaStream_t st) {
  KGE_REQUIRE(a.x && a.w && a.y && a.N > 0 && a.K > 0 && a.nz > 0, "linear_any: bad arguments");
  KGE_REQUIRE(a.act != ACT_EXP_DECAY || (a.act_coef && !a.w2), "linear_any: the decay needs its coefficients");
  if (a.T <= 0) return 0;
  if (linear_narrow_ok(a)) return a.N <= 8 ? launch_linear_narrow<1>(a, st) : a.N <= 16 ? launch_linear_narrow<2>(a, st) : launch_linear_narrow<4>(a, st);
  if (linear_few_ok(a)) return launch_linear_few(a, st);
  if (linear_short_ok(a)) {
    const size_t smem = (size_t)(WBM + WBN) * (a.K + MPAD) * 2;
    auto kern = a.act == ACT_SOFTPLUS ? linear_short_kernel<ACT_SOFTPLUS> : a.act == ACT_EXP_DECAY ? linear_short_kernel<ACT_EXP_DECAY> : linear_short_kernel<ACT_NONE>;
    KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (WBM + WBN) * (WMAXK + MPAD) * 2));      // for every K
    KGE_CUDA_OK(launch_pdl(kern, dim3((a.N + WBN - 1) / WBN, (a.T + WBM - 1) / WBM, a.nz), dim3(256), smem, st, a));
    return 0;
  }
  const int rows = a.group_off ? (a.max_rows > 0 ? a.max_rows : a.T) : a.T;
  dim3 grid((a.N + LBN - 1) / LBN, (rows + LBM - 1) / LBM, a.nz), block(256);
  KGE_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "linear_any: too many row tiles (%u) or slices (%u)", grid.y, grid.z);
  cudaError_t ce;
  const bool f32 = a.elt == KGE_ELT_F32;
  KGE_REQUIRE(!f32 || a.out_f32, "linear_any: float32 storage writes float32");
  if (f32) ce = a.w2 ? launch_pdl(linear_any_kernel<float, float, true>, grid, block, 0, st, a) : launch_pdl(linear_any_kernel<float, float, false>, grid, block, 0, st, a);
  else if (a.T <= 256 && a.K >= 256 && ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.w2)) & 15) == 0 && a.K % 8 == 0 && a.ldx % 8 == 0 &&
           a.x_zs % 8 == 0 && a.w_zs % 8 == 0) {
    if (a.w2) grid.x = (a.N + LBN / 2 - 1) / (LBN / 2);
    auto kern = a.out_f32 ? (a.w2 ? linear_stream_kernel<float, true> : linear_stream_kernel<float, false>)
                          : (a.w2 ? linear_stream_kernel<__nv_bfloat16, true> : linear_stream_kernel<__nv_bfloat16, false>);
    KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LINEAR_STREAM_SMEM));
    ce = launch_pdl(kern, grid, block, LINEAR_STREAM_SMEM, st, a);
  } else if (a.T <= 256) {       // few rows: the weights are the traffic
    if (a.out_f32) ce = a.w2 ? launch_pdl(linear_mma_kernel<float, true, 64>, grid, block, 0, st, a) : launch_pdl(linear_mma_kernel<float, false, 64>, grid, block, 0, st, a);
    else ce = a.w2 ? launch_pdl(linear_mma_kernel<__nv_bfloat16, true, 64>, grid, block, 0, st, a) : launch_pdl(linear_mma_kernel<__nv_bfloat16, false, 64>, grid, block, 0, st, a);
  } else if (a.out_f32) ce = a.w2 ? launch_pdl(linear_mma_kernel<float, true, 32>, grid, block, 0, st, a) : launch_pdl(linear_mma_kernel<float, false, 32>, grid, block, 0, st, a);
  else ce = a.w2 ? launch_pdl(linear_mma_kernel<__nv_bfloat16, true, 32>, grid, block, 0, st, a) : launch_pdl(linear_mma_kernel<__nv_bfloat16, false, 32>, grid, block, 0, st, a);
  KGE_CUDA_OK(ce);
  return 0;
}

// ------------------------------------------------------------------------------------------------ small row kernels
template <typename E, bool VEC>      // VEC: four columns per thread and pass (the rows of a step are a trip to memory each)
__global__ void embed_f32_kernel(float* res, const int32_t* ids, const E* table, int d) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const E* src = table + (int64_t)ids[t] * d;
  if (VEC) {
    for (int c = threadIdx.x * 4; c < d; c += blockDim.x * 4) {
      float v[4];
      ld4(src + c, v);
      st4(res + (int64_t)t * d + c, v);
    }
    return;
  }
  for (int c = threadIdx.x; c < d; c += blockDim.x) res[(int64_t)t * d + c] = ldf(src + c);
}
int embed_f32(float* res, const int32_t* ids, const void* table, int T, int d, int elt, cudaStream_t st) {
  if (T <= 0) return 0;
  const bool vec = d % 4 == 0 && ((reinterpret_cast<uintptr_t>(res) | reinterpret_cast<uintptr_t>(table)) & 15) == 0;
  const dim3 block(vec ? std::min(1024, (d / 4 + 31) / 32 * 32) : 128);
  cudaError_t ce;
  if (elt == KGE_ELT_F32) ce = vec ? launch_pdl(embed_f32_kernel<float, true>, dim3(T), block, 0, st, res, ids, (const float*)table, d) : launch_pdl(embed_f32_kernel<float, false>, dim3(T), block, 0, st, res, ids, (const float*)table, d);
  else ce = vec ? launch_pdl(embed_f32_kernel<__nv_bfloat16, true>, dim3(T), block, 0, st, res, ids, (const __nv_bfloat16*)table, d)
                : launch_pdl(embed_f32_kernel<__nv_bfloat16, false>, dim3(T), block, 0, st, res, ids, (const __nv_bfloat16*)table, d);
  KGE_CUDA_OK(ce);
  return 0;
}

// Ascending rows of three buffers to their front, in place.  A block has 32 pieces (16 bytes, or 2 where a row or a base is not a multiple of
// 16) of every row: it reads them all before it writes, so the time does not grow with the rows (turns of 16 in registers took 3.5 us for up
// to 16 rows and 7.7 for 30; 3.5 for one, 4.7 for 30 and 6 for 64 so).
struct FrontRows { uint8_t* p[3]; int64_t bytes[3]; };
template <class V>
__global__ void __launch_bounds__(256) rows_to_front_kernel(FrontRows f, const int32_t* rows, int n) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ uint4 front_sm[];
  V* held = reinterpret_cast<V*>(front_sm);                    // [n][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = f.bytes[blockIdx.y], pieces = row / (int64_t)sizeof(V), c = (int64_t)blockIdx.x * 32 + lane;
  if ((int64_t)blockIdx.x * 32 >= pieces) return;
  uint8_t* p = f.p[blockIdx.y] + c * (int64_t)sizeof(V);
  constexpr int U = 8, STEP = 256 / 32;
  for (int r0 = warp; r0 < n; r0 += U * STEP) {
    V v[U];
#pragma unroll
    for (int k = 0; k < U; ++k) if (c < pieces && r0 + k * STEP < n) v[k] = *reinterpret_cast<const V*>(p + rows[r0 + k * STEP] * row);
#pragma unroll
    for (int k = 0; k < U; ++k) if (c < pieces && r0 + k * STEP < n) held[(r0 + k * STEP) * 32 + lane] = v[k];
  }
  __syncthreads();
  for (int r = warp; r < n; r += STEP)
    if (c < pieces) *reinterpret_cast<V*>(p + r * row) = held[r * 32 + lane];
}
constexpr int FRONT_MAX = 256;
int rows_to_front(const int32_t* rows, int n, void* a, int64_t a_bytes, void* b, int64_t b_bytes, void* c, int64_t c_bytes, cudaStream_t st) {
  if (n <= 0) return 0;
  KGE_REQUIRE(n <= FRONT_MAX, "rows_to_front: %d rows", n);
  const FrontRows f = {{(uint8_t*)a, (uint8_t*)b, (uint8_t*)c}, {a_bytes, b_bytes, c_bytes}};
  const uintptr_t any = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)a_bytes | (uintptr_t)b_bytes | (uintptr_t)c_bytes;
  const int piece = (any & 15) == 0 ? 16 : 2;
  const dim3 grid((unsigned)((std::max(a_bytes, std::max(b_bytes, c_bytes)) / piece + 31) / 32), 3);
  const size_t smem = (size_t)n * 32 * piece;
  auto kern = piece == 16 ? rows_to_front_kernel<uint4> : rows_to_front_kernel<uint16_t>;
  if (smem > 48 * 1024) KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FRONT_MAX * 32 * 16));
  KGE_CUDA_OK(launch_pdl(kern, grid, dim3(256), smem, st, f, rows, n));
  return 0;
}

// one block per token; the row's four-column pieces when the tables allow
template <typename E, bool VEC>
__global__ void __launch_bounds__(256) embed_bigram_kernel(BigramArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, b = a.token_req[t], d = a.d, id = a.ids[t];
  int32_t* last = a.bigram ? reinterpret_cast<int32_t*>(a.state + (int64_t)a.slots[b] * a.slot_stride) : nullptr;
  int64_t row = a.buckets;
  if (a.bigram && a.positions[t] > 0) {
    const int64_t prev = t == a.qsl[b] ? *last : a.ids[t - 1];
    row = (prev * a.mul_prev + (int64_t)id * a.mul_cur) % a.buckets;
  }
  const E* e = (const E*)a.table + (int64_t)id * d;
  const E* g = (const E*)a.bigram + row * d;
  float* r = a.res + (int64_t)t * d;
  E* y = a.y ? (E*)a.y + (int64_t)t * d : nullptr;
  constexpr int W = VEC ? 4 : 1;
  for (int c = threadIdx.x * W; c < d; c += blockDim.x * W) {
    float u[4], v[4] = {0.f, 0.f, 0.f, 0.f};
    if (VEC) ld4(e + c, u); else u[0] = ldf(e + c);
    if (a.bigram) { if (VEC) ld4(g + c, v); else v[0] = ldf(g + c); }
#pragma unroll
    for (int k = 0; k < W; ++k) u[k] += v[k];
    if (VEC) { st4(r + c, u); if (y) st4(y + c, u); } else { r[c] = u[0]; if (y) stf(y + c, u[0]); }
  }
  if (a.bigram && a.inline_save) {
    __syncthreads();                            // every thread has read the slot
    if (threadIdx.x == 0) *last = id;
  }
}
__global__ void bigram_save_kernel(BigramArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < a.B && a.qsl[b + 1] > a.qsl[b]) *reinterpret_cast<int32_t*>(a.state + (int64_t)a.slots[b] * a.slot_stride) = a.ids[a.qsl[b + 1] - 1];
}
int embed_bigram(const BigramArgs& a, cudaStream_t st) {
  if (a.T <= 0) return 0;
  KGE_REQUIRE(a.table && (!a.bigram || (a.buckets > 0 && a.state)), "embed_bigram: bad arguments");
  const bool vec = a.d % 4 == 0 && ((reinterpret_cast<uintptr_t>(a.res) | reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.table) | reinterpret_cast<uintptr_t>(a.bigram)) & 15) == 0;
  cudaError_t ce;
  if (a.elt == KGE_ELT_F32) ce = vec ? launch_pdl(embed_bigram_kernel<float, true>, dim3(a.T), dim3(256), 0, st, a) : launch_pdl(embed_bigram_kernel<float, false>, dim3(a.T), dim3(256), 0, st, a);
  else ce = vec ? launch_pdl(embed_bigram_kernel<__nv_bfloat16, true>, dim3(a.T), dim3(256), 0, st, a) : launch_pdl(embed_bigram_kernel<__nv_bfloat16, false>, dim3(a.T), dim3(256), 0, st, a);
  KGE_CUDA_OK(ce);
  if (a.bigram && !a.inline_save) KGE_CUDA_OK(launch_pdl(bigram_save_kernel, dim3((a.B + 127) / 128), dim3(128), 0, st, a));
  return 0;
}

template <bool LN>      // rows of up to 8192 columns held in registers (defined with the layer norm below)
static bool norm_vec(void* y, const float* x, const int32_t* rows, const void* w, int R, int d, float eps, float offset, float out_scale, int elt, cudaStream_t st,
                     cudaError_t* ce);

template <typename E>
__global__ void rmsnorm_f32in_kernel(E* y, const float* x, const int32_t* rows, const E* w, int d, float eps, float offset, float out_scale) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[33];
  const int r = blockIdx.x;
  const float* src = x + (int64_t)(rows ? rows[r] : r) * d;
  float ss = 0.f;
  for (int c = threadIdx.x; c < d; c += blockDim.x) { const float v = src[c]; ss = fmaf(v, v, ss); }
  ss = block_sum(ss, red);
  const float inv = out_scale / sqrtf(ss / (float)d + eps);
  for (int c = threadIdx.x; c < d; c += blockDim.x) stf(y + (int64_t)r * d + c, src[c] * inv * (offset + ldf(w + c)));
}
int rmsnorm_f32in(void* y, const float* x, const int32_t* rows, const void* w, int R, int d, float eps, float offset, float out_scale, int elt,
                  cudaStream_t st) {
  if (R <= 0) return 0;
  cudaError_t ce;
  if (norm_vec<false>(y, x, rows, w, R, d, eps, offset, out_scale, elt, st, &ce)) { KGE_CUDA_OK(ce); return 0; }
  ce = elt == KGE_ELT_F32
      ? launch_pdl(rmsnorm_f32in_kernel<float>, dim3(R), dim3(256), 0, st, (float*)y, x, rows, (const float*)w, d, eps, offset, out_scale)
      : launch_pdl(rmsnorm_f32in_kernel<__nv_bfloat16>, dim3(R), dim3(256), 0, st, (__nv_bfloat16*)y, x, rows, (const __nv_bfloat16*)w, d, eps, offset, out_scale);
  KGE_CUDA_OK(ce);
  return 0;
}

// Both norms for rows of up to 8192 columns (a multiple of 4): the row is read once, as float4, and stays in registers for
// the statistics (layer norm: mean first, then the squared deviations) and the output (four values per store).
constexpr int NV_MAX = 8;
__device__ __forceinline__ float4 ldw4(const float* w) { return *reinterpret_cast<const float4*>(w); }
__device__ __forceinline__ float4 ldw4(const __nv_bfloat16* w) {
  const uint2 u = *reinterpret_cast<const uint2*>(w);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
__device__ __forceinline__ void st4(float* y, float4 v) { *reinterpret_cast<float4*>(y) = v; }
__device__ __forceinline__ void st4(__nv_bfloat16* y, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u; u.x = *reinterpret_cast<uint32_t*>(&a); u.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(y) = u;
}
template <typename E, bool LN>
__global__ void __launch_bounds__(256) norm_f32in_vec_kernel(E* y, const float* x, const int32_t* rows, const E* w, int d, float eps, float offset, float out_scale) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[33];
  const int r = blockIdx.x, nvec = d >> 2;
  const float* src = x + (int64_t)(rows ? rows[r] : r) * d;
  float4 v[NV_MAX];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV_MAX; ++i) {
    const int c = threadIdx.x + i * 256;
    v[i] = c < nvec ? *reinterpret_cast<const float4*>(src + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (LN) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
  }
  float mean = 0.f;
  if (LN) { mean = block_sum(s, red) / (float)d; __syncthreads(); }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV_MAX; ++i) {
    if (threadIdx.x + i * 256 < nvec) {
      v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
      ss = fmaf(v[i].x, v[i].x, ss); ss = fmaf(v[i].y, v[i].y, ss); ss = fmaf(v[i].z, v[i].z, ss); ss = fmaf(v[i].w, v[i].w, ss);
    }
  }
  ss = block_sum(ss, red);
  const float inv = out_scale / sqrtf(ss / (float)d + eps);
#pragma unroll
  for (int i = 0; i < NV_MAX; ++i) {
    const int c = threadIdx.x + i * 256;
    if (c < nvec) {
      const float4 g = ldw4(w + 4 * c);
      st4(y + (int64_t)r * d + 4 * c, make_float4(v[i].x * inv * (offset + g.x), v[i].y * inv * (offset + g.y), v[i].z * inv * (offset + g.z), v[i].w * inv * (offset + g.w)));
    }
  }
}
template <bool LN>
static bool norm_vec(void* y, const float* x, const int32_t* rows, const void* w, int R, int d, float eps, float offset, float out_scale, int elt, cudaStream_t st,
                     cudaError_t* ce) {
  if (d % 4 || d > 4 * 256 * NV_MAX || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(y) & 15) || (reinterpret_cast<uintptr_t>(w) & 15)) return false;
  *ce = elt == KGE_ELT_F32
      ? launch_pdl(norm_f32in_vec_kernel<float, LN>, dim3(R), dim3(256), 0, st, (float*)y, x, rows, (const float*)w, d, eps, offset, out_scale)
      : launch_pdl(norm_f32in_vec_kernel<__nv_bfloat16, LN>, dim3(R), dim3(256), 0, st, (__nv_bfloat16*)y, x, rows, (const __nv_bfloat16*)w, d, eps, offset, out_scale);
  return true;
}

// weight-only layer norm of an fp32 row: mean first, then the mean of the squared deviations (no cancellation)
template <typename E>
__global__ void layernorm_f32in_kernel(E* y, const float* x, const int32_t* rows, const E* w, int d, float eps, float out_scale) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[33];
  const int r = blockIdx.x;
  const float* src = x + (int64_t)(rows ? rows[r] : r) * d;
  float s = 0.f;
  for (int c = threadIdx.x; c < d; c += blockDim.x) s += src[c];
  const float mean = block_sum(s, red) / (float)d;
  __syncthreads();
  float ss = 0.f;
  for (int c = threadIdx.x; c < d; c += blockDim.x) { const float v = src[c] - mean; ss = fmaf(v, v, ss); }
  ss = block_sum(ss, red);
  const float inv = out_scale / sqrtf(ss / (float)d + eps);
  for (int c = threadIdx.x; c < d; c += blockDim.x) stf(y + (int64_t)r * d + c, (src[c] - mean) * inv * ldf(w + c));
}
int layernorm_f32in(void* y, const float* x, const int32_t* rows, const void* w, int R, int d, float eps, float out_scale, int elt, cudaStream_t st) {
  if (R <= 0) return 0;
  cudaError_t ce;
  if (norm_vec<true>(y, x, rows, w, R, d, eps, 0.f, out_scale, elt, st, &ce)) { KGE_CUDA_OK(ce); return 0; }
  ce = elt == KGE_ELT_F32
      ? launch_pdl(layernorm_f32in_kernel<float>, dim3(R), dim3(256), 0, st, (float*)y, x, rows, (const float*)w, d, eps, out_scale)
      : launch_pdl(layernorm_f32in_kernel<__nv_bfloat16>, dim3(R), dim3(256), 0, st, (__nv_bfloat16*)y, x, rows, (const __nv_bfloat16*)w, d, eps, out_scale);
  KGE_CUDA_OK(ce);
  return 0;
}

template <typename E>
__global__ void residual_combine_kernel(float* res, CombineArgs a, int64_t n, int d) {
  pdl_launch_dependents();
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / d; const int c = (int)(i % d);
    float s = 0.f;
    for (int k = 0; k < a.n; ++k) {
      const float f = a.rscale[k] ? a.scale[k] * a.rscale[k][t * a.rs_stride[k]] : a.scale[k];
      s = fmaf(f, ldf((const E*)a.src[k] + t * a.ld[k] + c), s);
    }
    res[i] += s;
  }
}
// four columns per thread: one float4 of the stream, one 8- or 16-byte piece of every source
template <typename E>
__global__ void residual_combine_vec_kernel(float* res, CombineArgs a, int64_t n4, int d4) {
  pdl_launch_dependents();
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / d4; const int c = (int)(i % d4) * 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < a.n; ++k) {
      const float f = a.rscale[k] ? a.scale[k] * a.rscale[k][t * a.rs_stride[k]] : a.scale[k];
      const float4 v = ldw4((const E*)a.src[k] + t * a.ld[k] + c);
      s.x = fmaf(f, v.x, s.x); s.y = fmaf(f, v.y, s.y); s.z = fmaf(f, v.z, s.z); s.w = fmaf(f, v.w, s.w);
    }
    float4* dst = reinterpret_cast<float4*>(res) + i;
    float4 o = *dst;
    o.x += s.x; o.y += s.y; o.z += s.z; o.w += s.w;
    *dst = o;
  }
}
int residual_combine(float* res, const CombineArgs& a, int T, int d, int elt, cudaStream_t st) {
  if (T <= 0 || a.n <= 0) return 0;
  const int64_t n = (int64_t)T * d;
  bool vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(res) & 15) == 0;
  for (int k = 0; k < a.n; ++k) vec = vec && a.ld[k] % 4 == 0 && (reinterpret_cast<uintptr_t>(a.src[k]) & 15) == 0;
  if (vec) {
    const int grid4 = (int)std::min<int64_t>((n / 4 + 255) / 256, 148 * 16);
    cudaError_t ce4 = elt == KGE_ELT_F32 ? launch_pdl(residual_combine_vec_kernel<float>, dim3(grid4), dim3(256), 0, st, res, a, n / 4, d / 4)
                                         : launch_pdl(residual_combine_vec_kernel<__nv_bfloat16>, dim3(grid4), dim3(256), 0, st, res, a, n / 4, d / 4);
    KGE_CUDA_OK(ce4);
    return 0;
  }
  const int grid = (int)std::min<int64_t>((n + 255) / 256, 148 * 8);
  cudaError_t ce = elt == KGE_ELT_F32 ? launch_pdl(residual_combine_kernel<float>, dim3(grid), dim3(256), 0, st, res, a, n, d)
                                      : launch_pdl(residual_combine_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, st, res, a, n, d);
  KGE_CUDA_OK(ce);
  return 0;
}

// The sum above and the next sublayer's norm of the new row in one pass: the row stays in registers, so it is not read back, and the loads of
// all sources are under way together.  The same arithmetic as residual_combine and norm_f32in_vec_kernel one after the other.
// NV: four-column pieces per thread.  2312 rows of 2048, one to four sources: 36 us in two launches, 16 here.
template <typename E, bool LN, int NV>
__global__ void __launch_bounds__(256) combine_norm_kernel(float* res, CombineArgs a, E* y, const E* w, int d, float eps, float offset) {
  pdl_launch_dependents();
  __shared__ float red[33];
  const int64_t t = blockIdx.x;
  const int nvec = d >> 2;
  float4 g[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * 256;
    if (c < nvec) g[i] = ldw4(w + 4 * c);
  }
  pdl_wait();
  float4* row = reinterpret_cast<float4*>(res + t * d);
  float4 v[NV], src[4][NV];
  float f[4];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * 256;
    v[i] = c < nvec ? row[c] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < a.n && c < nvec) src[k][i] = ldw4((const E*)a.src[k] + t * a.ld[k] + 4 * c);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) f[k] = k < a.n ? (a.rscale[k] ? a.scale[k] * a.rscale[k][t * a.rs_stride[k]] : a.scale[k]) : 0.f;
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * 256;
    if (c < nvec) {
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < a.n) {
          const float4 x = src[k][i];
          o.x = fmaf(f[k], x.x, o.x); o.y = fmaf(f[k], x.y, o.y); o.z = fmaf(f[k], x.z, o.z); o.w = fmaf(f[k], x.w, o.w);
        }
      v[i].x += o.x; v[i].y += o.y; v[i].z += o.z; v[i].w += o.w;
      row[c] = v[i];
    }
    if (LN) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
  }
  float mean = 0.f;
  if (LN) { mean = block_sum(s, red) / (float)d; __syncthreads(); }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (threadIdx.x + i * 256 < nvec) {
      v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
      ss = fmaf(v[i].x, v[i].x, ss); ss = fmaf(v[i].y, v[i].y, ss); ss = fmaf(v[i].z, v[i].z, ss); ss = fmaf(v[i].w, v[i].w, ss);
    }
  ss = block_sum(ss, red);
  const float inv = 1.f / sqrtf(ss / (float)d + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = threadIdx.x + i * 256;
    if (c < nvec)
      st4(y + t * d + 4 * c, make_float4(v[i].x * inv * (offset + g[i].x), v[i].y * inv * (offset + g[i].y), v[i].z * inv * (offset + g[i].z), v[i].w * inv * (offset + g[i].w)));
  }
}
template <typename E, bool LN>
static cudaError_t launch_combine_norm(float* res, const CombineArgs& a, void* y, const void* w, int T, int d, float eps, float offset, cudaStream_t st) {
  auto kern = d <= 1024 ? combine_norm_kernel<E, LN, 1> : d <= 2048 ? combine_norm_kernel<E, LN, 2> : combine_norm_kernel<E, LN, 4>;
  return launch_pdl(kern, dim3(T), dim3(256), 0, st, res, a, (E*)y, (const E*)w, d, eps, offset);
}
bool combine_norm_ok(const float* res, const CombineArgs& a, const void* y, const void* w, int d) {
  bool ok = a.n > 0 && d % 4 == 0 && d <= 4096 && ((reinterpret_cast<uintptr_t>(res) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
  for (int k = 0; k < a.n; ++k) ok = ok && a.ld[k] % 4 == 0 && (reinterpret_cast<uintptr_t>(a.src[k]) & 15) == 0;
  return ok;
}
int combine_norm(float* res, const CombineArgs& a, void* y, const void* w, int T, int d, float eps, bool layer_norm, int elt, cudaStream_t st) {
  KGE_REQUIRE(combine_norm_ok(res, a, y, w, d), "combine_norm: sizes");
  if (T <= 0) return 0;
  // RMS weights apply as 1 + w, those of the layer norm as they are
  KGE_CUDA_OK(elt == KGE_ELT_F32 ? (layer_norm ? launch_combine_norm<float, true>(res, a, y, w, T, d, eps, 0.f, st) : launch_combine_norm<float, false>(res, a, y, w, T, d, eps, 1.f, st))
                                 : (layer_norm ? launch_combine_norm<__nv_bfloat16, true>(res, a, y, w, T, d, eps, 0.f, st) : launch_combine_norm<__nv_bfloat16, false>(res, a, y, w, T, d, eps, 1.f, st)));
  return 0;
}

__global__ void logits_to_elt16_kernel(uint16_t* out, const float* in, int R, int V, int ld, bool f16) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t n = (int64_t)R * V;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / V; const int c = (int)(i % V);
    out[r * ld + c] = f16 ? __half_as_ushort(__float2half_rn(in[i])) : __bfloat16_as_ushort(__float2bfloat16_rn(in[i]));
  }
}
int logits_to_elt16(void* out, const float* in, int R, int V, int ld_out, bool f16, cudaStream_t st) {
  if (R <= 0) return 0;
  const int grid = (int)std::min<int64_t>(((int64_t)R * V + 255) / 256, 148 * 8);
  KGE_CUDA_OK(launch_pdl(logits_to_elt16_kernel, dim3(grid), dim3(256), 0, st, (uint16_t*)out, in, R, V, ld_out, f16));
  return 0;
}

__global__ void elt16_to_f32_kernel(float* out, const __nv_bfloat16* in, int64_t n) {
  pdl_launch_dependents();
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) out[i] = __bfloat162float(in[i]);
}
int elt16_to_f32(float* out, const void* in_bf16, int64_t n, cudaStream_t st) {
  if (n <= 0) return 0;
  KGE_CUDA_OK(launch_pdl(elt16_to_f32_kernel, dim3((unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8)), dim3(256), 0, st, out, (const __nv_bfloat16*)in_bf16, n));
  return 0;
}


__device__ __forceinline__ float softcap_f(float v, float cap) { return cap * tanhf(v / cap); }
__global__ void softcap_rows_kernel(float* l32, __nv_bfloat16* l16, int R, int V, int ld16, float cap) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t n = (int64_t)R * V;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / V; const int c = (int)(i % V);
    const float v = softcap_f(l16 ? __bfloat162float(l16[r * ld16 + c]) : l32[i], cap);
    if (l32) l32[i] = v;
    if (l16) l16[r * ld16 + c] = __float2bfloat16_rn(v);
  }
}
int softcap_rows(float* l32, void* l16, int R, int V, int ld16, float cap, cudaStream_t st) {
  if (R <= 0 || cap <= 0.f) return 0;
  const int grid = (int)std::min<int64_t>(((int64_t)R * V + 255) / 256, 148 * 8);
  KGE_CUDA_OK(launch_pdl(softcap_rows_kernel, dim3(grid), dim3(256), 0, st, l32, (__nv_bfloat16*)l16, R, V, ld16, cap));
  return 0;
}

}  // namespace kge
