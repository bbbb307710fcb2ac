// Recurrent token mixers with per-request state slots, in bfloat16 or float32 storage and fp32 state:
//   - the gated linear recurrence (RG-LRU): causal per-channel convolution whose last inputs are carried in the slot,
//     then S <- a S + sqrt(1 - a^2) i u with a = exp(-c r softplus(lam)), one thread per (request, channel);
//   - the matrix memory (mLSTM) with a running maximum that starts at 0, one block per (request, head), the dim x vdim
//     state in shared memory, one thread per value column.
// A request whose first row of the step is position 0 starts from zero; otherwise from what its slot holds.  Rows of a
// request are processed in order, so cutting a prompt into steps anywhere gives the same arithmetic.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "elt_access.cuh"
#include "gate_math.cuh"
#include "hybrid_ops.h"

namespace kge {

constexpr int MAX_TAPS = 16;

template <typename E>
__global__ void rglru_conv_kernel(RglruArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int b = a.token_req[t], pos = a.positions[t], rs = a.qsl[b];
  const int p0 = a.positions[rs];                         // position of the request's first row in this step
  const E* yx = (const E*)a.yx;
  const float* tail = a.state + (int64_t)a.slots[b] * a.slot_stride + a.width;
  for (int c = threadIdx.x; c < a.width; c += blockDim.x) {
    float acc = ldf((const E*)a.conv_b + c);
    for (int j = 0; j < a.taps; ++j) {
      const int back = a.taps - 1 - j, sp = pos - back;
      float xv = 0.f;
      if (sp >= p0) xv = ldf(yx + (int64_t)(t - back) * 2 * a.width + a.width + c);
      else if (sp >= 0) xv = tail[(int64_t)(sp - p0 + a.taps - 1) * a.width + c];
      acc = fmaf(ldf((const E*)a.conv_w + (int64_t)c * a.taps + j), xv, acc);
    }
    stf((E*)a.u + (int64_t)t * a.width + c, acc);
  }
}

// The same for bfloat16 rows in 16-byte pieces: a thread takes eight channels of four tokens, so that all its loads (taps x tokens,
// and the taps' weights once) are in flight together.  Same order of summation.  2312 tokens x 2560 by 4 taps: 20 us (28 with
// the taps' weights one by one, 43 with a channel per thread and pass), 2 tokens: 8.6 us (11, 27).
// TAPS 4: a channel's taps lie side by side, so those of eight channels are 64 bytes, read (like the bias) before the wait; 0: any number.
constexpr int RC_TOK = 4;
template <int TAPS>
__global__ void __launch_bounds__(128) rglru_conv_vec_kernel(RglruArgs a) {
  pdl_launch_dependents();
  const int c = (blockIdx.y * 128 + threadIdx.x) * 8, t0 = blockIdx.x * RC_TOK;
  if (c >= a.width) return;
  const int taps = TAPS ? TAPS : a.taps;
  uint4 wq[TAPS ? TAPS : 1];
#pragma unroll
  for (int i = 0; i < TAPS; ++i) wq[i] = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.conv_w + (int64_t)c * TAPS + i * 8);
  const __nv_bfloat16* yx = (const __nv_bfloat16*)a.yx + a.width + c;
  float acc[RC_TOK][8], bias[8];
  int back_rows[RC_TOK], back_pos[RC_TOK], p0s[RC_TOK];
  const float* tails[RC_TOK];
  {
    const uint4 v = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.conv_b + c);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) bias[i] = (i & 1) ? bf_hi(w[i / 2]) : bf_lo(w[i / 2]);
  }
  pdl_wait();
#pragma unroll
  for (int k = 0; k < RC_TOK; ++k) {
    const int t = min(t0 + k, a.T - 1), b = a.token_req[t], rs = a.qsl[b];
    p0s[k] = a.positions[rs];
    back_pos[k] = a.positions[t];
    back_rows[k] = t;
    tails[k] = a.state + (int64_t)a.slots[b] * a.slot_stride + a.width + c;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[k][i] = bias[i];
  }
#pragma unroll 4
  for (int j = 0; j < taps; ++j) {
    const int back = taps - 1 - j;
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (TAPS) {
        const uint32_t q[4] = {wq[(i * TAPS + j) / 8 % (TAPS ? TAPS : 1)].x, wq[(i * TAPS + j) / 8 % (TAPS ? TAPS : 1)].y, wq[(i * TAPS + j) / 8 % (TAPS ? TAPS : 1)].z, wq[(i * TAPS + j) / 8 % (TAPS ? TAPS : 1)].w};
        const uint32_t pair = q[(i * TAPS + j) % 8 / 2];
        w[i] = (j & 1) ? bf_hi(pair) : bf_lo(pair);
      } else {
        w[i] = ldf((const __nv_bfloat16*)a.conv_w + (int64_t)(c + i) * taps + j);
      }
    }
#pragma unroll
    for (int k = 0; k < RC_TOK; ++k) {
      const int sp = back_pos[k] - back;
      float x[8];
      if (sp >= p0s[k]) {
        const uint4 v = *reinterpret_cast<const uint4*>(yx + (int64_t)(back_rows[k] - back) * 2 * a.width);
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = (i & 1) ? bf_hi(u[i / 2]) : bf_lo(u[i / 2]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = sp >= 0 ? tails[k][(int64_t)(sp - p0s[k] + taps - 1) * a.width + i] : 0.f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[k][i] = fmaf(w[i], x[i], acc[k][i]);
    }
  }
#pragma unroll
  for (int k = 0; k < RC_TOK; ++k)
    if (t0 + k < a.T)
      *reinterpret_cast<uint4*>((__nv_bfloat16*)a.u + (int64_t)(t0 + k) * a.width + c) =
          make_uint4(pack_bf2(acc[k][0], acc[k][1]), pack_bf2(acc[k][2], acc[k][3]), pack_bf2(acc[k][4], acc[k][5]), pack_bf2(acc[k][6], acc[k][7]));
}

int rglru_conv(const RglruArgs& a, cudaStream_t st) {
  if (a.T <= 0) return 0;
  KGE_REQUIRE(a.taps >= 1 && a.taps <= MAX_TAPS, "rglru_conv: %d taps (1..%d)", a.taps, MAX_TAPS);
  // few rows of few channels leave its threads a chain of loads each where the other kernel has a thread for every channel (64 rows of
  // 64 channels 5.1 us here and 2.6 there, of 264 5.6 and 3.6; 64 of 1024 6.3 and 6.1, 256 of 1024 6.4 and 7.0, 2312 of 64 4.3 and 4.7)
  if (a.elt == KGE_ELT_BF16 && (a.width >= 1024 || a.T > 1024) && a.width % 8 == 0 && ((reinterpret_cast<uintptr_t>(a.yx) | reinterpret_cast<uintptr_t>(a.u) | reinterpret_cast<uintptr_t>(a.conv_b)) & 15) == 0) {
    auto kern = a.taps == 4 && (reinterpret_cast<uintptr_t>(a.conv_w) & 15) == 0 ? rglru_conv_vec_kernel<4> : rglru_conv_vec_kernel<0>;
    KGE_CUDA_OK(launch_pdl(kern, dim3((a.T + RC_TOK - 1) / RC_TOK, (a.width / 8 + 127) / 128), dim3(128), 0, st, a));
    return 0;
  }
  cudaError_t ce = a.elt == KGE_ELT_F32 ? launch_pdl(rglru_conv_kernel<float>, dim3(a.T), dim3(256), 0, st, a)
                                        : launch_pdl(rglru_conv_kernel<__nv_bfloat16>, dim3(a.T), dim3(256), 0, st, a);
  KGE_CUDA_OK(ce);
  return 0;
}

__device__ __forceinline__ float sigmoidf_(float v) { return 1.f / (1.f + expf(-v)); }
__device__ __forceinline__ float gelu_tanhf_(float v) { return 0.5f * v * (1.f + tanhf(0.79788456080286536f * (v + 0.044715f * v * v * v))); }

template <typename E>
__global__ void __launch_bounds__(128) rglru_scan_kernel(RglruArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= a.width) return;
  const int rs = a.qsl[b], re = a.qsl[b + 1], p0 = a.positions[rs], n = re - rs;
  float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride;
  const E* yx = (const E*)a.yx;
  const E* u = (const E*)a.u;
  E* out = (E*)a.out;
  const float sp = a.decay_c * softplusf_(ldf((const E*)a.lam + c));
  float S = p0 > 0 ? slot[c] : 0.f;
  // eight tokens at a time: all their operands are requested before the first is used, so the recurrence itself - one
  // dependent fma per token - is what the loop waits for, not a memory round trip per token
  constexpr int G = 8;
  for (int t0 = rs; t0 < re; t0 += G) {
    float gr[G], gi[G], uv[G], yv[G];
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int t = min(t0 + k, re - 1);
      gr[k] = a.gates[(int64_t)t * 2 * a.width + c];
      gi[k] = a.gates[(int64_t)t * 2 * a.width + a.width + c];
      uv[k] = ldf(u + (int64_t)t * a.width + c);
      yv[k] = ldf(yx + (int64_t)t * 2 * a.width + c);
    }
#pragma unroll
    for (int k = 0; k < G; ++k) {
      if (t0 + k < re) {
        const float r = sigmoidf_(gr[k]), i = sigmoidf_(gi[k]);
        const float log_a = -sp * r;
        const float av = expf(log_a);
        const float mult = sqrtf(-expm1f(2.f * log_a));          // sqrt(1 - a^2) without cancellation near a = 1
        S = fmaf(av, S, mult * i * uv[k]);
        stf(out + (int64_t)(t0 + k) * a.width + c, S * gelu_tanhf_(yv[k]));
      }
    }
  }
  slot[c] = S;
  // the conv's next inputs: positions p1 - (taps - 1) .. p1 - 1 with p1 = p0 + n, from this step's rows or the old tail
  float nt[MAX_TAPS];
  float* tail = slot + a.width;
#pragma unroll
  for (int k = 0; k < MAX_TAPS; ++k) {
    if (k >= a.taps - 1) break;
    const int sp2 = p0 + n - (a.taps - 1) + k;
    float v = 0.f;
    if (sp2 >= p0) v = ldf(yx + (int64_t)(rs + sp2 - p0) * 2 * a.width + a.width + c);
    else if (sp2 >= 0) v = tail[(int64_t)(sp2 - p0 + a.taps - 1) * a.width + c];
    nt[k] = v;
  }
#pragma unroll
  for (int k = 0; k < MAX_TAPS; ++k) {
    if (k >= a.taps - 1) break;
    tail[(int64_t)k * a.width + c] = nt[k];
  }
}

int rglru_scan(const RglruArgs& a, cudaStream_t st) {
  if (a.T <= 0 || a.B <= 0) return 0;
  KGE_REQUIRE(a.taps >= 1 && a.taps <= MAX_TAPS, "rglru_scan: %d taps (1..%d)", a.taps, MAX_TAPS);
  const dim3 grid(a.B, (a.width + 127) / 128), block(128);
  if (a.T > a.B) {                       // some request brings several rows
    const int rc = rglru_coefficients(a, st);
    return rc ? rc : rglru_walk(a, st);
  }
  cudaError_t ce = a.elt == KGE_ELT_F32 ? launch_pdl(rglru_scan_kernel<float>, grid, block, 0, st, a)
                                        : launch_pdl(rglru_scan_kernel<__nv_bfloat16>, grid, block, 0, st, a);
  KGE_CUDA_OK(ce);
  return 0;
}

// ------------------------------------------------------------------------------------------------ matrix memory
template <typename E>
__global__ void mlstm_step_kernel(MlstmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float sm[];
  const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int dim = a.dim, vdim = a.vdim;
  float* S = sm;                       // [dim][vdim]
  float* nv = S + (int64_t)dim * vdim; // [dim]
  float* ks = nv + dim;                // [dim]
  float* qs = ks + dim;                // [dim]
  float* red = qs + dim;               // [33]
  const int rs = a.qsl[b], re = a.qsl[b + 1], p0 = a.positions[rs];
  float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride + (int64_t)h * ((int64_t)dim * vdim + dim + 1);
  const bool fresh = p0 == 0;
  for (int i = tid; i < dim * vdim + dim; i += blockDim.x) S[i] = fresh ? 0.f : slot[i];     // S then n: contiguous in both
  float m = fresh ? 0.f : slot[(int64_t)dim * vdim + dim];
  __syncthreads();
  const E *qp = (const E*)a.q, *kp = (const E*)a.k, *vp = (const E*)a.v, *gp = (const E*)a.g;
  const float nw = tid < vdim ? ldf((const E*)a.norm_w + h * vdim + tid) : 0.f;
  for (int t = rs; t < re; ++t) {
    if (tid < dim) {
      ks[tid] = ldf(kp + (int64_t)t * a.ld + h * dim + tid);
      qs[tid] = ldf(qp + (int64_t)t * a.ld + h * dim + tid) * a.q_scale;
    }
    const float ip = a.gates[(int64_t)t * 2 * a.H + h], fp = a.gates[(int64_t)t * 2 * a.H + a.H + h];
    const float it = a.cap * tanhf(ip / a.cap);
    const float fc = a.cap * tanhf(fp / a.cap);
    const float ft = fminf(fc, 0.f) - log1pf(expf(-fabsf(fc)));          // logsigmoid
    const float mn = fmaxf(ft + m, it);
    const float fa = expf(ft + m - mn), ia = expf(it - mn);
    m = mn;
    __syncthreads();
    float part = 0.f;
    if (tid < dim) {
      const float nn = fmaf(fa, nv[tid], ia * ks[tid]);
      nv[tid] = nn;
      part = nn * qs[tid];
    }
    const float nq = block_sum(part, red);
    float o = 0.f;
    if (tid < vdim) {
      const float vv = ia * ldf(vp + (int64_t)t * a.ld + h * vdim + tid);
      float num = 0.f;
      for (int d = 0; d < dim; ++d) {
        const float s = fmaf(fa, S[d * vdim + tid], ks[d] * vv);
        S[d * vdim + tid] = s;
        num = fmaf(s, qs[d], num);
      }
      o = num / (fmaxf(fabsf(nq), expf(-m)) + a.den_eps);
    }
    const float ss = block_sum(o * o, red);
    if (tid < vdim) {
      const float inv = 1.f / sqrtf(ss / (float)vdim + a.eps);
      const float gate = 1.f / (1.f + expf(-ldf(gp + (int64_t)t * a.ld + h * vdim + tid)));
      stf((E*)a.out + (int64_t)t * a.ldo + h * vdim + tid, o * inv * nw * gate * a.out_scale);
    }
  }
  __syncthreads();
  for (int i = tid; i < dim * vdim + dim; i += blockDim.x) slot[i] = S[i];
  if (tid == 0) slot[(int64_t)dim * vdim + dim] = m;
}

// The same recurrence with a head's value columns split over blocks of 64 threads: a thread keeps its column of the
// state in registers (dim <= 128), the first warp keeps the normaliser n, and the un-normalised read-out goes to an fp32
// scratch; mlstm_norm_gate_kernel then divides each head by its root mean square and applies weight and output gate.
// All blocks of a head read n and m at their start, and not all blocks of a launch start together: the block that has the new
// ones leaves them in scratch, and the second kernel, which runs when all blocks are done, puts them into the state.
// More blocks than (request, head) pairs fill the machine when few requests prefill, and the state never sits in shared memory.
constexpr int ML_MAXD = 128, ML_COLS = 64, ML_THREADS = ML_COLS + 32;      // two warps of value columns, one for the normaliser

// gate pre-activations -> log gates, in place, for every token at once (the recurrence then needs two exponentials a token)
__global__ void mlstm_log_gates_kernel(float* gates, int T, int H, float cap) {
  pdl_launch_dependents();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * 2 * H) return;
  const float c = cap * tanhf(gates[i] / cap);
  gates[i] = (i % (2 * H)) < H ? c : fminf(c, 0.f) - log1pf(expf(-fabsf(c)));     // input gate | logsigmoid for the forget gate
}

template <typename E>
__global__ void __launch_bounds__(ML_THREADS) mlstm_cols_kernel(MlstmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ __align__(16) float ks[ML_MAXD], qs[ML_MAXD], nv[ML_MAXD];
  __shared__ float nq_s;
  const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, c = blockIdx.z * ML_COLS + tid;
  const int dim = a.dim, vdim = a.vdim;
  const bool colw = tid < ML_COLS;                 // a value-column thread (the last warp keeps n instead)
  const bool col = colw && c < vdim;
  const int rs = a.qsl[b], re = a.qsl[b + 1], p0 = a.positions[rs];
  float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride + (int64_t)h * ((int64_t)dim * vdim + dim + 1);
  const bool fresh = p0 == 0;
  float S[ML_MAXD];
#pragma unroll
  for (int d = 0; d < ML_MAXD; ++d) S[d] = (d < dim && col && !fresh) ? slot[(int64_t)d * vdim + c] : 0.f;
  for (int d = tid; d < ML_MAXD; d += ML_THREADS) { nv[d] = (d < dim && !fresh) ? slot[(int64_t)dim * vdim + d] : 0.f; ks[d] = 0.f; qs[d] = 0.f; }
  float m = fresh ? 0.f : slot[(int64_t)dim * vdim + dim];
  const E *qp = (const E*)a.q, *kp = (const E*)a.k, *vp = (const E*)a.v;
  __syncthreads();
  // operands of the NEXT token are requested while the current one is computed (two key / query entries per thread)
  float kn[2], qn[2], vn, ipn, fpn;
  auto fetch = [&](int t) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int d = tid + j * ML_COLS;
      kn[j] = (colw && d < dim) ? ldf(kp + (int64_t)t * a.ld + h * dim + d) : 0.f;
      qn[j] = (colw && d < dim) ? ldf(qp + (int64_t)t * a.ld + h * dim + d) * a.q_scale : 0.f;
    }
    vn = col ? ldf(vp + (int64_t)t * a.ld + h * vdim + c) : 0.f;
    ipn = a.gates[(int64_t)t * 2 * a.H + h];
    fpn = a.gates[(int64_t)t * 2 * a.H + a.H + h];
  };
  if (rs < re) fetch(rs);
  for (int t = rs; t < re; ++t) {
    if (colw) { ks[tid] = kn[0]; ks[tid + ML_COLS] = kn[1]; qs[tid] = qn[0]; qs[tid + ML_COLS] = qn[1]; }
    const float it = ipn, ft = fpn, vcur = vn;     // log gates (mlstm_log_gates_kernel ran before)
    if (t + 1 < re) fetch(t + 1);
    const float mn = fmaxf(ft + m, it);
    const float fa = expf(ft + m - mn), ia = expf(it - mn);
    m = mn;
    const float vv = ia * vcur;
    __syncthreads();
    float num = 0.f;
    if (!colw) {
      const int ln = tid - ML_COLS;
      float part = 0.f;
      for (int d = ln; d < dim; d += 32) {
        const float nn = fmaf(fa, nv[d], ia * ks[d]);
        nv[d] = nn;
        part = fmaf(nn, qs[d], part);
      }
      part = warp_sum(part);
      if (ln == 0) nq_s = part;
    } else {
      float n0 = 0.f, n1 = 0.f, n2 = 0.f, n3 = 0.f;       // four chains: the read-out does not wait on one long dependency
#pragma unroll
      for (int d4 = 0; d4 < ML_MAXD / 4; ++d4) {
        if (d4 * 4 < dim) {                      // dim is a multiple of 4 on this path
          const float4 k4 = reinterpret_cast<const float4*>(ks)[d4], q4 = reinterpret_cast<const float4*>(qs)[d4];
          S[d4 * 4 + 0] = fmaf(fa, S[d4 * 4 + 0], k4.x * vv); n0 = fmaf(S[d4 * 4 + 0], q4.x, n0);
          S[d4 * 4 + 1] = fmaf(fa, S[d4 * 4 + 1], k4.y * vv); n1 = fmaf(S[d4 * 4 + 1], q4.y, n1);
          S[d4 * 4 + 2] = fmaf(fa, S[d4 * 4 + 2], k4.z * vv); n2 = fmaf(S[d4 * 4 + 2], q4.z, n2);
          S[d4 * 4 + 3] = fmaf(fa, S[d4 * 4 + 3], k4.w * vv); n3 = fmaf(S[d4 * 4 + 3], q4.w, n3);
        }
      }
      num = (n0 + n1) + (n2 + n3);
    }
    __syncthreads();
    if (col) a.o_scratch[(int64_t)t * a.H * vdim + h * vdim + c] = num / (fmaxf(fabsf(nq_s), expf(-m)) + a.den_eps);
  }
  if (col) {
#pragma unroll
    for (int d = 0; d < ML_MAXD; ++d) if (d < dim) slot[(int64_t)d * vdim + c] = S[d];
  }
  if (blockIdx.z == 0) {
    __syncthreads();
    float* nm = a.nm_scratch + ((int64_t)b * a.H + h) * (dim + 1);
    for (int d = tid; d < dim; d += ML_THREADS) nm[d] = nv[d];
    if (tid == 0) nm[dim] = m;
  }
}

// Prompts: the same recurrence evaluated 32 tokens at a time (chunkwise form), all in fp32.  With b_t the running sum of
// the log forget gates inside the chunk and (C, n, m) the state before it,
//   m_t = max(b_t + m, max_{s<=t}(b_t - b_s + i_s))                     (equal to the step-by-step maximum)
//   num_t = e^(b_t + m - m_t) C^T q_t + sum_{s<=t} e^(b_t - b_s + i_s - m_t) (q_t . k_s) v_s
//   n_t . q_t likewise with n and the same weights;   C' = e^(b_L + m - m_L) C + sum_s e^(b_L - b_s + i_s - m_L) k_s v_s^T
// so a token costs the same multiply-adds as one recurrence step but the 32 tokens of a chunk are independent: no
// barrier and no dependent chain per token.  A thread still owns one value column of C in registers.
constexpr int ML_CH = 32, ML_NSL = 4, ML_DS = ML_MAXD / ML_NSL;      // tokens per chunk; key-dimension slices per column; dims per slice
constexpr int MC_COLS = 32;          // value columns per block of the chunkwise kernel: more, smaller blocks fill the machine when few requests prefill

// Block = 32 value columns x 4 slices of the key dimension (128 threads): a thread keeps C[its 32 dims][its column] in
// registers, so the read-out and the update of a chunk are spread over four warps; the slices' partial read-outs meet in
// shared memory and are summed in slice order.
template <typename E>
__global__ void __launch_bounds__(MC_COLS * ML_NSL) mlstm_chunk_kernel(MlstmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float csm[];
  constexpr int NT = MC_COLS * ML_NSL;
  const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, ct = tid % MC_COLS, sl = tid / MC_COLS, c = blockIdx.z * MC_COLS + ct;
  const int dim = a.dim, vdim = a.vdim, d0 = sl * ML_DS;
  float* qs = csm;                           // [ML_CH][dim]   q_t * q_scale
  float* ks = qs + ML_CH * dim;              // [ML_CH][dim]   k_s, later u_s * k_s
  float* Sw = ks + ML_CH * dim;              // [ML_CH][ML_CH] weighted scores (s <= t)
  float* nv = Sw + ML_CH * ML_CH;            // [ML_MAXD]
  float* li = nv + ML_MAXD;                  // [ML_CH] log input gate
  float* bc = li + ML_CH;                    // [ML_CH] running sum of log forget gates
  float* mt = bc + ML_CH;                    // [ML_CH] running maximum
  float* nq = mt + ML_CH;                    // [ML_CH] n . q_t (state part)
  float* us = nq + ML_CH;                    // [ML_CH] weight of token s in the state after the chunk
  float* vs = us + ML_CH;                    // [ML_CH][MC_COLS] this block's value columns of the chunk's tokens
  float* part = vs + ML_CH * MC_COLS;        // [ML_NSL][ML_CH][MC_COLS] partial read-outs of the slices
  const bool col = c < vdim;
  const int rs = a.qsl[b], re = a.qsl[b + 1], p0 = a.positions[rs];
  float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride + (int64_t)h * ((int64_t)dim * vdim + dim + 1);
  const bool fresh = p0 == 0;
  float C[ML_DS];
#pragma unroll
  for (int d = 0; d < ML_DS; ++d) C[d] = (d0 + d < dim && col && !fresh) ? slot[(int64_t)(d0 + d) * vdim + c] : 0.f;
  for (int d = tid; d < ML_MAXD; d += NT) nv[d] = (d < dim && !fresh) ? slot[(int64_t)dim * vdim + d] : 0.f;
  float m = fresh ? 0.f : slot[(int64_t)dim * vdim + dim];
  const E *qp = (const E*)a.q, *kp = (const E*)a.k, *vp = (const E*)a.v;
  for (int t0 = rs; t0 < re; t0 += ML_CH) {
    const int L = min(ML_CH, re - t0);
    __syncthreads();                                         // the previous chunk's shared arrays are no longer read
    for (int i = tid; i < L * dim; i += NT) {
      const int t = i / dim, d = i % dim;
      qs[i] = ldf(qp + (int64_t)(t0 + t) * a.ld + h * dim + d) * a.q_scale;
      ks[i] = ldf(kp + (int64_t)(t0 + t) * a.ld + h * dim + d);
    }
    for (int i = tid; i < L * MC_COLS; i += NT) {
      const int s2 = i / MC_COLS, cc = blockIdx.z * MC_COLS + i % MC_COLS;
      vs[i] = cc < vdim ? ldf(vp + (int64_t)(t0 + s2) * a.ld + h * vdim + cc) : 0.f;
    }
    if (tid == 0) {                                          // the chunk's gate scalars: 32 short steps
      float run = 0.f, mm = m;
      for (int t = 0; t < L; ++t) {
        const float it = a.gates[(int64_t)(t0 + t) * 2 * a.H + h], ft = a.gates[(int64_t)(t0 + t) * 2 * a.H + a.H + h];
        mm = fmaxf(ft + mm, it);
        run += ft;
        li[t] = it; bc[t] = run; mt[t] = mm;
      }
    }
    __syncthreads();
    const float bL = bc[L - 1], mL = mt[L - 1];
    // weighted scores Sw[t][s] = e^(b_t - b_s + i_s - m_t) (q_t . k_s) for s <= t; the state part of n . q_t; the tokens' weights in the new state
    for (int i = tid; i < L * L; i += NT) {
      const int t = i / L, s2 = i % L;
      float w = 0.f;
      if (s2 <= t) {
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
        for (int d4 = 0; d4 < dim / 4; ++d4) {
          const float4 q4 = reinterpret_cast<const float4*>(qs + t * dim)[d4], k4 = reinterpret_cast<const float4*>(ks + s2 * dim)[d4];
          a0 = fmaf(q4.x, k4.x, a0); a1 = fmaf(q4.y, k4.y, a1); a2 = fmaf(q4.z, k4.z, a2); a3 = fmaf(q4.w, k4.w, a3);
        }
        w = expf(bc[t] - bc[s2] + li[s2] - mt[t]) * ((a0 + a1) + (a2 + a3));
      }
      Sw[t * ML_CH + s2] = w;
    }
    for (int t = tid; t < L; t += NT) {
      float acc = 0.f;
      for (int d = 0; d < dim; ++d) acc = fmaf(nv[d], qs[t * dim + d], acc);
      nq[t] = acc;
      us[t] = expf(bL - bc[t] + li[t] - mL);
    }
    // this slice's part of C^T q_t for every token of the chunk
    for (int t = 0; t < L; ++t) {
      float n0 = 0.f, n1 = 0.f, n2 = 0.f, n3 = 0.f;
#pragma unroll
      for (int d4 = 0; d4 < ML_DS / 4; ++d4) {
        if (d0 + d4 * 4 < dim) {
          const float4 q4 = reinterpret_cast<const float4*>(qs + t * dim + d0)[d4];
          n0 = fmaf(C[d4 * 4 + 0], q4.x, n0); n1 = fmaf(C[d4 * 4 + 1], q4.y, n1);
          n2 = fmaf(C[d4 * 4 + 2], q4.z, n2); n3 = fmaf(C[d4 * 4 + 3], q4.w, n3);
        }
      }
      part[(sl * ML_CH + t) * MC_COLS + ct] = (n0 + n1) + (n2 + n3);
    }
    __syncthreads();
    // tokens t = sl, sl + 4, ...: slices summed in order, the chunk's own tokens added, normaliser, out
    for (int t = sl; t < L; t += ML_NSL) {
      float inter = 0.f;
#pragma unroll
      for (int k = 0; k < ML_NSL; ++k) inter += part[(k * ML_CH + t) * MC_COLS + ct];
      float intra = 0.f, rowsum = 0.f;
      for (int s2 = 0; s2 <= t; ++s2) { const float w = Sw[t * ML_CH + s2]; intra = fmaf(w, vs[s2 * MC_COLS + ct], intra); rowsum += w; }
      const float g = expf(bc[t] + m - mt[t]);
      const float num = fmaf(g, inter, intra);
      const float den = fmaxf(fabsf(fmaf(g, nq[t], rowsum)), expf(-mt[t])) + a.den_eps;
      if (col) a.o_scratch[(int64_t)(t0 + t) * a.H * vdim + h * vdim + c] = num / den;
    }
    // state after the chunk: C' = G C + sum_s u_s k_s v_s^T with G = e^(b_L + m - m_L); n likewise
    const float G = expf(bL + m - mL);
#pragma unroll
    for (int d = 0; d < ML_DS; ++d) C[d] *= G;
    for (int s2 = 0; s2 < L; ++s2) {
      const float x = us[s2] * vs[s2 * MC_COLS + ct];
#pragma unroll
      for (int d4 = 0; d4 < ML_DS / 4; ++d4) {
        if (d0 + d4 * 4 < dim) {
          const float4 k4 = reinterpret_cast<const float4*>(ks + s2 * dim + d0)[d4];
          C[d4 * 4 + 0] = fmaf(k4.x, x, C[d4 * 4 + 0]); C[d4 * 4 + 1] = fmaf(k4.y, x, C[d4 * 4 + 1]);
          C[d4 * 4 + 2] = fmaf(k4.z, x, C[d4 * 4 + 2]); C[d4 * 4 + 3] = fmaf(k4.w, x, C[d4 * 4 + 3]);
        }
      }
    }
    for (int d = tid; d < dim; d += NT) {
      float acc = G * nv[d];
      for (int s2 = 0; s2 < L; ++s2) acc = fmaf(us[s2], ks[s2 * dim + d], acc);
      nv[d] = acc;
    }
    m = mL;
  }
  __syncthreads();
  if (col) {
#pragma unroll
    for (int d = 0; d < ML_DS; ++d) if (d0 + d < dim) slot[(int64_t)(d0 + d) * vdim + c] = C[d];
  }
  if (blockIdx.z == 0) {                                       // see mlstm_cols_kernel
    float* nm = a.nm_scratch + ((int64_t)b * a.H + h) * (dim + 1);
    for (int d = tid; d < dim; d += NT) nm[d] = nv[d];
    if (tid == 0) nm[dim] = m;
  }
}

// The same chunkwise form for bfloat16 operands on mma.sync tensor cores, 64 tokens at a time.  Block = one (request, head) and
// 32 value columns; the columns of C stay in fp32 accumulators of the eight warps (16 key dimensions each) from the first chunk
// to the last.  q, k and v are bfloat16 already; what is fp32 (C, the weighted scores, the weighted values) enters a product as
// three bfloat16 terms that add up to its 24 bits, so every product is exact to fp32 and sums are fp32; a chunk's update is
// summed by itself and then joined to C by one fma.  A chunk costs four barriers and ~250 MMAs per warp; the next chunk's
// rows arrive by cp.async meanwhile.
// What bounds it: mma.sync, 32 cycles a quarter of an SM for 16 x 8 x 16 numbers, in the chain of a request's chunks: 7.5 us each.  Where
// that leaves SMs without work (2 requests x 4 heads x 8 column blocks), up to eight blocks share a head's columns: each goes over all
// chunks before its own with the updates of the state alone (a third of the work, the same numbers in every block) and reads out its own,
// whose run is the shorter the more lies before it; the last writes the state.  Nothing is exchanged.  us with one block and so: prompts of
// 1150 and 1162 tokens, 4 heads of 128 x 256 (two blocks) 150 / 102, one of 1300 (four) 157 / 79, of 4096 471 / 229, of 129 27 / 19.  The
// head's column blocks, which formed a cluster because of n and m, are free of each other: 4 x 1024 tokens 252 / 142.
// Prompts of 1150 and 1162 tokens: error against 64 bits 1.0e-6 of the read-out and 2.5e-7 of the state (the fp32 kernel above, 1101 us,
// 1.5e-6 and 5.0e-7); one prompt of 1300 with a state before it: 6.6e-7 and 1.1e-7 (7.5e-7 and 2.3e-7).
// A request with one row of the step takes a plain path on the same block (fp32, one pass over its columns).
constexpr float MM_SHARE = 0.65f;      // a run of chunks beside the one before it
constexpr int MM_CH = 64, MM_COLS = 32, MM_THREADS = 256, MM_LDQ = 128 + 8, MM_LDV = MM_COLS + 8;
struct MlstmTile {
  __nv_bfloat16 q[2][MM_CH][MM_LDQ], k[2][MM_CH][MM_LDQ], v[2][MM_CH][MM_LDV];
  __nv_bfloat16 x[3][MM_CH][MM_LDV];            // u_s v_s in three terms
  __nv_bfloat16 c[3][128][MM_LDV];              // C before the chunk in three terms
  float out[MM_CH][MM_COLS + 2], rows[MM_CH];   // the second key half's part of the read-out and of the weights' sum
  float nv[128], nsum[2][128], nq[MM_CH];
  float2 e[MM_CH], M[MM_CH];                    // i_s - b_s and m_t - b_t, each as a sum of two
  float floor_[MM_CH], us[MM_CH], gt[MM_CH];    // e^(-m_t); weights of the tokens and of C in the new state
  float G;
};

__device__ __forceinline__ void ml_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ml_ldsm(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ml_ldsm_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
// (lo, hi) as three packed pairs of bfloat16 whose sums are the fp32 values
__device__ __forceinline__ void ml_split(float lo, float hi, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = pack_bf2(lo, hi);
    lo -= bf_lo(t[i]); hi -= bf_hi(t[i]);
  }
}

template <bool SHARED>
__global__ void __launch_bounds__(MM_THREADS) mlstm_mma_kernel(MlstmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  typedef __nv_bfloat16 E;
  extern __shared__ __align__(16) unsigned char mm_raw[];
  MlstmTile& sm = *reinterpret_cast<MlstmTile*>(mm_raw);
  // ranks of a cluster share a head's columns of a request: rank r has the read-outs of the r-th run of chunks
  const int S = SHARED ? (int)cluster_nctarank() : 1, rank = SHARED ? (int)cluster_ctarank() : 0, b = blockIdx.x / S, h = blockIdx.y, c0 = blockIdx.z * MM_COLS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int dim = a.dim, vdim = a.vdim, H = a.H;
  const int rs = a.qsl[b], re = a.qsl[b + 1];
  if (re <= rs) return;
  const int p0 = a.positions[rs];
  float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride + (int64_t)h * ((int64_t)dim * vdim + dim + 1);
  const bool fresh = p0 == 0;
  const E *qp = (const E*)a.q + h * dim, *kp = (const E*)a.k + h * dim, *vp = (const E*)a.v + h * vdim + c0;
  const int ncol = min(MM_COLS, vdim - c0);
  const float m0 = fresh ? 0.f : slot[(int64_t)dim * vdim + dim];
  for (int d = tid; d < 128; d += MM_THREADS) sm.nv[d] = d < dim && !fresh ? slot[(int64_t)dim * vdim + d] : 0.f;
  __syncthreads();

  float* nm = a.nm_scratch + ((int64_t)b * H + h) * (dim + 1);
  if (re - rs == 1) {
    if (rank + 1 < S) return;
    // one token: thread = (column, eighth of the key dimensions)
    const int col = lane, per = (dim + 7) / 8, d0 = warp * per, d1 = min(dim, d0 + per);
    const float it = a.gates[(int64_t)rs * 2 * H + h], ft = a.gates[(int64_t)rs * 2 * H + H + h];
    const float mn = fmaxf(ft + m0, it), fa = expf(ft + m0 - mn), ia = expf(it - mn);
    float* qs = &sm.out[0][0]; float* ks = qs + 128;
    for (int d = tid; d < dim; d += MM_THREADS) { qs[d] = ldf(qp + (int64_t)rs * a.ld + d) * a.q_scale; ks[d] = ldf(kp + (int64_t)rs * a.ld + d); }
    const float vv = col < ncol ? ia * ldf(vp + (int64_t)rs * a.ld + col) : 0.f;
    __syncthreads();
    float num = 0.f;
    if (col < ncol)
#pragma unroll 8
      for (int d = d0; d < d1; ++d) {
        float* s = slot + (int64_t)d * vdim + c0 + col;
        const float n = fmaf(fa, fresh ? 0.f : *s, ks[d] * vv);
        *s = n;
        num = fmaf(n, qs[d], num);
      }
    float* part = &sm.out[16][0];                              // [8][32]
    part[warp * 32 + col] = num;
    float np = 0.f;
    for (int d = tid; d < dim; d += MM_THREADS) {
      const float n = fmaf(fa, sm.nv[d], ia * ks[d]);
      sm.nv[d] = n;
      np = fmaf(n, qs[d], np);
    }
    np = warp_sum(np);
    if (lane == 0) sm.nq[warp] = np;
    __syncthreads();
    if (warp == 0 && col < ncol) {
      float o = 0.f, nq = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) { o += part[w * 32 + col]; nq += sm.nq[w]; }
      a.o_scratch[(int64_t)rs * H * vdim + h * vdim + c0 + col] = o / (fmaxf(fabsf(nq), expf(-mn)) + a.den_eps);
    }
    if (blockIdx.z == 0) {
      for (int d = tid; d < dim; d += MM_THREADS) nm[d] = sm.nv[d];
      if (tid == 0) nm[dim] = mn;
    }
    return;
  }

  const int mt0 = warp * 16;                                   // this warp's key dimensions of C
  const bool has_c = mt0 < dim;
  float C[MM_COLS / 8][4];
  auto write_terms = [&]() {
#pragma unroll
    for (int n = 0; n < MM_COLS / 8; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t t[3];
        ml_split(C[n][2 * r], C[n][2 * r + 1], t);
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(&sm.c[i][mt0 + g + 8 * r][n * 8 + t4 * 2]) = t[i];
      }
  };
#pragma unroll
  for (int n = 0; n < MM_COLS / 8; ++n)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int d = mt0 + g + 8 * (q >> 1), col = n * 8 + t4 * 2 + (q & 1);
      C[n][q] = d < dim && col < ncol && !fresh ? slot[(int64_t)d * vdim + c0 + col] : 0.f;
    }
  if (SHARED) cluster_arrive();                                      // the last rank writes the state back when all have read it
  // the rank's run: [own0, own1), each MM_SHARE of the one before it, since what lies before a run costs its rank the updates only
  const int chunks = (re - rs + MM_CH - 1) / MM_CH;
  auto border = [&](int r) {
    float before = 0.f, all = 0.f, w = 1.f;
    for (int i = 0; i < S; ++i, w *= MM_SHARE) { all += w; if (i < r) before += w; }
    return r >= S ? re : min(re, rs + MM_CH * (int)(chunks * (before / all) + 0.5f));
  };
  const int own0 = SHARED ? border(rank) : rs, own1 = SHARED ? border(rank + 1) : re;
  const bool last = !SHARED || rank + 1 == S;
  if (!SHARED || own0 == rs) write_terms();

  // rows of 64 tokens: q and k in 16-byte pieces (dim / 8 per row), v likewise (the host checked the alignment)
  const int pieces = dim / 8;
  auto copy16 = [&](void* dst, const E* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(in ? src : qp), "r"(in ? 16u : 0u) : "memory");
  };
  auto fetch = [&](int t0, int st) {
    const bool full = !SHARED || t0 >= own0;                   // no read-out: no q
    for (int i = tid; i < MM_CH * pieces; i += MM_THREADS) {
      const int r = i / pieces, c = (i - r * pieces) * 8;
      const bool in = t0 + r < re;
      if (full) copy16(&sm.q[st][r][c], qp + (int64_t)(t0 + r) * a.ld + c, in);
      copy16(&sm.k[st][r][c], kp + (int64_t)(t0 + r) * a.ld + c, in);
    }
    const int r = tid >> 2, c = (tid & 3) * 8;
    copy16(&sm.v[st][r][c], vp + (int64_t)(t0 + r) * a.ld + c, t0 + r < re && c < ncol);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int rg = (warp & 3) * 16, half = warp >> 2;            // this warp's 16 tokens; its half of the keys / key dimensions
  const int ksteps = dim / 16, kh = (ksteps + 1) / 2, k_begin = half ? kh : 0, k_end = half ? ksteps : kh;
  double m = m0;                                               // (warp 0) the running maximum before the chunk
  const int end = last ? re : own0 < own1 ? own1 : rs;         // (a rank without a run has nothing to do)
  if (rs < end) fetch(rs, 0);
  int st = 0;
  for (int t0 = rs; t0 < end; t0 += MM_CH, st ^= 1) {
    const bool full = !SHARED || t0 >= own0;
    // the gate scalars of the chunk, two tokens per lane of the first warp: with e_s = i_s - b_s and M_t = max(m, max_{s<=t} e_s),
    // m_t = b_t + M_t, and the weights above are e^(m - M_t) and e^(e_s - M_t)
    float it[2], ft[2];
    if (warp == 0) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = t0 + 2 * lane + j;
        it[j] = t < re ? a.gates[(int64_t)t * 2 * H + h] : -INFINITY;
        ft[j] = t < re ? a.gates[(int64_t)t * 2 * H + H + h] : 0.f;
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                           // the chunk's rows and C's terms are there; the other stage is free
    if (t0 + MM_CH < end) fetch(t0 + MM_CH, st ^ 1);
    if (warp == 0) {
      // running sums in 64 bits: b_t grows with the chunk, and what the weights need are differences
      const double pair = (double)ft[0] + (double)ft[1];
      double run = pair;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const double v = __shfl_up_sync(0xffffffffu, run, o); if (lane >= o) run += v; }
      const double b1 = run, b0 = run - pair + (double)ft[0];
      const double e0 = (double)it[0] - b0, e1 = (double)it[1] - b1;
      double mx = fmax(e0, e1);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const double v = __shfl_up_sync(0xffffffffu, mx, o); if (lane >= o) mx = fmax(mx, v); }
      double before = __shfl_up_sync(0xffffffffu, mx, 1);
      before = lane == 0 ? m : fmax(before, m);
      const double M0 = fmax(before, e0), M1 = fmax(M0, e1);
      const double bL = __shfl_sync(0xffffffffu, b1, 31), ML = __shfl_sync(0xffffffffu, M1, 31);
      const int i0 = 2 * lane, i1 = i0 + 1;
      auto two = [](double v) { const float hi = (float)v; return make_float2(hi, hi == -INFINITY ? 0.f : (float)(v - (double)hi)); };
      sm.e[i0] = two(e0); sm.e[i1] = two(e1); sm.M[i0] = two(M0); sm.M[i1] = two(M1);
      sm.floor_[i0] = expf(-(float)(b0 + M0)); sm.floor_[i1] = expf(-(float)(b1 + M1));
      sm.us[i0] = expf((float)(e0 - ML)); sm.us[i1] = expf((float)(e1 - ML));
      sm.gt[i0] = expf((float)(m - M0)); sm.gt[i1] = expf((float)(m - M1));
      if (lane == 0) sm.G = expf((float)(m - ML));
      m = bL + ML;
    }
    // q_t . k_s for this warp's tokens and its half of the keys (none where all keys lie behind the tokens)
    const bool keys = full && half * 32 <= rg + 15;
    float sc[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
    float in[MM_COLS / 8][4], ia[MM_COLS / 8][4];              // state part and chunk part of the read-out
#pragma unroll
    for (int n = 0; n < MM_COLS / 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) in[n][q] = ia[n][q] = 0.f;
    for (int k = 0; k < (full ? ksteps : 0); ++k) {
      uint32_t af[4];
      const bool mine = k >= k_begin && k < k_end;
      if (!keys && !mine) continue;
      ml_ldsm(af, &sm.q[st][rg + (lane & 15)][k * 16 + (lane >> 4) * 8]);
      if (keys)
#pragma unroll
        for (int n2 = 0; n2 < 2; ++n2) {
          uint32_t bf[4];
          ml_ldsm(bf, &sm.k[st][half * 32 + n2 * 16 + (lane & 7) + ((lane >> 4) & 1) * 8][k * 16 + ((lane >> 3) & 1) * 8]);
          // each step's sums start from zero and join by a rounded addition: the tensor core's own accumulation truncates, and a
          // token whose normaliser cancels shows it
          float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
          ml_mma(s0, af, bf[0], bf[1]);
          ml_mma(s1, af, bf[2], bf[3]);
#pragma unroll
          for (int q = 0; q < 4; ++q) { sc[2 * n2][q] += s0[q]; sc[2 * n2 + 1][q] += s1[q]; }
        }
      if (mine)                                                // C^T q_t over this warp's half of the key dimensions
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int n2 = 0; n2 < MM_COLS / 16; ++n2) {
            uint32_t bf[4];
            ml_ldsm_t(bf, &sm.c[i][k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][n2 * 16 + (lane >> 4) * 8]);
            ml_mma(in[2 * n2], af, bf[0], bf[1]);
            ml_mma(in[2 * n2 + 1], af, bf[2], bf[3]);
          }
    }
    if (full) {
      // n . q_t, four threads per token
      const int tok = tid >> 2;
      float acc = 0.f;
      for (int d = (tid & 3) * 2; d < dim; d += 8) {
        const uint32_t u = *reinterpret_cast<const uint32_t*>(&sm.q[st][tok][d]);
        acc = fmaf(sm.nv[d], bf_lo(u), acc); acc = fmaf(sm.nv[d + 1], bf_hi(u), acc);
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      if ((tid & 3) == 0) sm.nq[tok] = acc * a.q_scale;
    }
    __syncthreads();                                           // the gate scalars are there
    {
      // the tokens' weighted values, in three terms, and their keys' weighted sum
      const int r = tid >> 2, c = (tid & 3) * 8;
      const float u = sm.us[r];
      const uint4 v = *reinterpret_cast<const uint4*>(&sm.v[st][r][c]);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      uint32_t o[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t t[3];
        ml_split(u * bf_lo(w[j]), u * bf_hi(w[j]), t);
        o[0][j] = t[0]; o[1][j] = t[1]; o[2][j] = t[2];
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(&sm.x[i][r][c]) = make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
      const int d = tid & 127, s0 = (tid >> 7) * 32;
      float acc = 0.f;
      if (d < dim)
#pragma unroll 8
        for (int s2 = s0; s2 < s0 + 32; ++s2) acc = fmaf(sm.us[s2], __bfloat162float(sm.k[st][s2][d]), acc);
      sm.nsum[tid >> 7][d] = acc;
    }
    float rowsum[2] = {0.f, 0.f};
    if (keys) {
      uint32_t wt[2][3][4];                                    // weights as A fragments, [16 keys][term]
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int tok = rg + g + 8 * r, key = half * 32 + n * 8 + t4 * 2;
          const float2 M = sm.M[tok];
          float w[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float2 e = sm.e[key + j];
            w[j] = key + j <= tok ? expf((e.x - M.x) + (e.y - M.y)) * (sc[n][2 * r + j] * a.q_scale) : 0.f;
            rowsum[r] += w[j];
          }
          uint32_t t[3];
          ml_split(w[0], w[1], t);
#pragma unroll
          for (int i = 0; i < 3; ++i) wt[n >> 1][i][(n & 1) * 2 + r] = t[i];
        }
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int n2 = 0; n2 < MM_COLS / 16; ++n2) {
          uint32_t bf[4];
          ml_ldsm_t(bf, &sm.v[st][half * 32 + k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][n2 * 16 + (lane >> 4) * 8]);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            ml_mma(ia[2 * n2], wt[k][i], bf[0], bf[1]);
            ml_mma(ia[2 * n2 + 1], wt[k][i], bf[2], bf[3]);
          }
        }
    }
    float num[MM_COLS / 8][4];
    if (full) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      rowsum[r] += __shfl_xor_sync(0xffffffffu, rowsum[r], 1);
      rowsum[r] += __shfl_xor_sync(0xffffffffu, rowsum[r], 2);
    }
#pragma unroll
    for (int n = 0; n < MM_COLS / 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) num[n][q] = fmaf(sm.gt[rg + g + 8 * (q >> 1)], in[n][q] * a.q_scale, ia[n][q]);
    if (half) {
#pragma unroll
      for (int n = 0; n < MM_COLS / 8; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r)
          *reinterpret_cast<float2*>(&sm.out[rg + g + 8 * r][n * 8 + t4 * 2]) = make_float2(num[n][2 * r], num[n][2 * r + 1]);
      if (t4 == 0) { sm.rows[rg + g] = rowsum[0]; sm.rows[rg + g + 8] = rowsum[1]; }
    }
    }
    __syncthreads();                                           // all have read C's terms; x, the sums and the halves are there
    if (full && !half) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int tok = rg + g + 8 * r, t = t0 + tok;
        if (t < re) {
          const float den = fmaxf(fabsf(fmaf(sm.gt[tok], sm.nq[tok], rowsum[r] + sm.rows[tok])), sm.floor_[tok]) + a.den_eps;
          float* o = a.o_scratch + (int64_t)t * H * vdim + h * vdim + c0;
#pragma unroll
          for (int n = 0; n < MM_COLS / 8; ++n) {
            const float2 o2 = *reinterpret_cast<const float2*>(&sm.out[tok][n * 8 + t4 * 2]);
            const int col = n * 8 + t4 * 2;
            if (col < ncol) o[col] = (num[n][2 * r] + o2.x) / den;
            if (col + 1 < ncol) o[col + 1] = (num[n][2 * r + 1] + o2.y) / den;
          }
        }
      }
    }
    if (!last && t0 + MM_CH >= end) break;                     // the state is another rank's to go on with
    // C' = G C + k^T x
    const float G = sm.G;
    if (has_c) {
      float D[MM_COLS / 8][4];
#pragma unroll
      for (int n = 0; n < MM_COLS / 8; ++n) D[n][0] = D[n][1] = D[n][2] = D[n][3] = 0.f;
#pragma unroll
      for (int k = 0; k < MM_CH / 16; ++k) {
        uint32_t af[4];
        ml_ldsm_t(af, &sm.k[st][k * 16 + (lane & 7) + (lane >> 4) * 8][mt0 + ((lane >> 3) & 1) * 8]);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int n2 = 0; n2 < MM_COLS / 16; ++n2) {
            uint32_t bf[4];
            ml_ldsm_t(bf, &sm.x[i][k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][n2 * 16 + (lane >> 4) * 8]);
            ml_mma(D[2 * n2], af, bf[0], bf[1]);
            ml_mma(D[2 * n2 + 1], af, bf[2], bf[3]);
          }
      }
#pragma unroll
      for (int n = 0; n < MM_COLS / 8; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) C[n][q] = fmaf(G, C[n][q], D[n][q]);
      if (!SHARED || t0 + MM_CH >= own0) write_terms();
    }
    if (tid < 128) sm.nv[tid] = fmaf(G, sm.nv[tid], sm.nsum[0][tid] + sm.nsum[1][tid]);
  }
  if (SHARED) cluster_wait();
  if (!last) return;
  if (has_c) {
#pragma unroll
    for (int n = 0; n < MM_COLS / 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int d = mt0 + g + 8 * (q >> 1), col = n * 8 + t4 * 2 + (q & 1);
        if (col < ncol) slot[(int64_t)d * vdim + c0 + col] = C[n][q];
      }
  }
  if (blockIdx.z == 0) {
    if (tid < dim) nm[tid] = sm.nv[tid];           // its own entry of the last update
    if (tid == 0) nm[dim] = (float)m;
  }
}

// n and m, dim + 1 numbers, by n threads: five at a time, since loads do not pass stores by themselves
__device__ __forceinline__ void ml_copy_nm(float* slot, const float* nm, int dim, int i, int n) {
  for (; i <= dim; i += 5 * n) {
    float v[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) if (i + k * n <= dim) v[k] = nm[i + k * n];
#pragma unroll
    for (int k = 0; k < 5; ++k) if (i + k * n <= dim) slot[i + k * n] = v[k];
  }
}
template <typename E>
__global__ void mlstm_norm_gate_kernel(MlstmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[33];
  const int t = blockIdx.x, h = blockIdx.y;
  if (t >= a.T) {                                              // blocks beyond the tokens: a request's new n and m
    const int b = t - a.T;
    const float* nm = a.nm_scratch + ((int64_t)b * a.H + h) * (a.dim + 1);
    float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride + ((int64_t)h + 1) * ((int64_t)a.dim * a.vdim + a.dim + 1) - (a.dim + 1);
    ml_copy_nm(slot, nm, a.dim, threadIdx.x, blockDim.x);
    return;
  }
  const float* o = a.o_scratch + (int64_t)t * a.H * a.vdim + h * a.vdim;
  float ss = 0.f;
  for (int c = threadIdx.x; c < a.vdim; c += blockDim.x) ss = fmaf(o[c], o[c], ss);
  ss = block_sum(ss, red);
  const float inv = a.out_scale / sqrtf(ss / (float)a.vdim + a.eps);
  for (int c = threadIdx.x; c < a.vdim; c += blockDim.x) {
    const float gate = 1.f / (1.f + expf(-ldf((const E*)a.g + (int64_t)t * a.ld + h * a.vdim + c)));
    stf((E*)a.out + (int64_t)t * a.ldo + h * a.vdim + c, o[c] * inv * ldf((const E*)a.norm_w + h * a.vdim + c) * gate);
  }
}

// The same for 16-bit rows in 16-byte pieces, a warp per (token, head) and NV pieces a lane: no barrier, and all of a row's loads at once.
// 2312 tokens, 4 heads of 256 values: 20 us above and 8 here (cold caches).
template <int NV>
__global__ void __launch_bounds__(256) mlstm_norm_gate_wide_kernel(MlstmArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  typedef __nv_bfloat16 E;
  const int lane = threadIdx.x & 31, vdim = a.vdim;
  const int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int t = (int)(item / a.H), h = (int)(item - (int64_t)t * a.H);
  if (t >= a.T) {                                              // behind the tokens: a request's new n and m
    const int b = t - a.T;
    if (b >= a.B) return;
    const float* nm = a.nm_scratch + ((int64_t)b * a.H + h) * (a.dim + 1);
    float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride + ((int64_t)h + 1) * ((int64_t)a.dim * vdim + a.dim + 1) - (a.dim + 1);
    ml_copy_nm(slot, nm, a.dim, lane, 32);
    return;
  }
  const float* o = a.o_scratch + ((int64_t)t * a.H + h) * vdim;
  float4 v[NV][2];
  uint4 g[NV], w[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int c = (lane + j * 32) * 8;
    v[j][0] = v[j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < vdim) {
      v[j][0] = *reinterpret_cast<const float4*>(o + c); v[j][1] = *reinterpret_cast<const float4*>(o + c + 4);
      g[j] = *reinterpret_cast<const uint4*>((const E*)a.g + (int64_t)t * a.ld + h * vdim + c);
      w[j] = *reinterpret_cast<const uint4*>((const E*)a.norm_w + h * vdim + c);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) { const float4 q = v[j][i]; ss = fmaf(q.x, q.x, ss); ss = fmaf(q.y, q.y, ss); ss = fmaf(q.z, q.z, ss); ss = fmaf(q.w, q.w, ss); }
  const float inv = a.out_scale / sqrtf(warp_sum(ss) / (float)vdim + a.eps);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int c = (lane + j * 32) * 8;
    if (c >= vdim) continue;
    const float x[8] = {v[j][0].x, v[j][0].y, v[j][0].z, v[j][0].w, v[j][1].x, v[j][1].y, v[j][1].z, v[j][1].w};
    const uint32_t gu[4] = {g[j].x, g[j].y, g[j].z, g[j].w}, wu[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float g0 = 1.f / (1.f + expf(-bf_lo(gu[i]))), g1 = 1.f / (1.f + expf(-bf_hi(gu[i])));
      r[i] = pack_bf2(x[2 * i] * inv * bf_lo(wu[i]) * g0, x[2 * i + 1] * inv * bf_hi(wu[i]) * g1);
    }
    *reinterpret_cast<uint4*>((E*)a.out + (int64_t)t * a.ldo + h * vdim + c) = make_uint4(r[0], r[1], r[2], r[3]);
  }
}
// bfloat16 rows: the kernel above where pieces of 16 bytes are aligned and there is more than the SMs hold in blocks of 256 threads at once (one
// prompt of 100 tokens and 4 heads of 256, the whole chunkwise form: 16.7 us with a block a row, 17.2 with a warp; 4096 tokens 145 and 124;
// 200 single tokens, 8 heads of 64, the whole step 27.3 and 28.5)
static int mlstm_norm_gate(const MlstmArgs& a, dim3 grid, int threads, cudaStream_t st) {
  const bool wide = (int64_t)a.T * a.H * a.vdim > 8 * 148 * 256 && a.vdim % 8 == 0 && a.vdim <= 1024 && a.ld % 8 == 0 && a.ldo % 8 == 0 &&
                    ((reinterpret_cast<uintptr_t>(a.o_scratch) | reinterpret_cast<uintptr_t>(a.g) | reinterpret_cast<uintptr_t>(a.norm_w) | reinterpret_cast<uintptr_t>(a.out)) & 15) == 0;
  const dim3 wgrid((unsigned)(((int64_t)(a.T + a.B) * a.H + 7) / 8));
  if (!wide) KGE_CUDA_OK(launch_pdl(mlstm_norm_gate_kernel<__nv_bfloat16>, grid, dim3(threads), 0, st, a));
  else KGE_CUDA_OK(launch_pdl(a.vdim <= 256 ? mlstm_norm_gate_wide_kernel<1> : a.vdim <= 512 ? mlstm_norm_gate_wide_kernel<2> : mlstm_norm_gate_wide_kernel<4>, wgrid, dim3(256), 0, st, a));
  return 0;
}

// Decode steps, one row a request, in one launch: log gates, state, read-out, its norm over the head and the output gate.  A block has 32
// value columns of a head, a warp 16 of the key dimensions (DIM / 8); the blocks of a head form a cluster, which adds up the head's
// squares and holds the new normaliser back until all have read the old one.  4 heads of 128 x 256, us back to back (cold caches), in
// three launches (mlstm_log_gates, mlstm_cols, mlstm_norm_gate) and here: 1 request 12.5 (18.5) and 4.0 (10.3), 2 requests 12.5 and 4.2,
// 8 requests 13.4 and 6.4, 64 requests 25.0 and 21.6, 200 requests 75.3 and 63.5 (HBM: the state is read and written).
template <typename E>
__global__ void __launch_bounds__(256) mlstm_token_kernel(MlstmArgs a) {
  cluster_arrive_relaxed();                                    // waited for before the first remote store
  pdl_launch_dependents();
  __shared__ __align__(16) float qs[ML_MAXD], ks[ML_MAXD], part[8][33], np_s[8], squares[8];
  const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = blockIdx.z * 32 + lane;
  const int dim = a.dim, vdim = a.vdim, per = (dim + 7) / 8, d0 = warp * per, d1 = min(dim, d0 + per);
  // slots, positions and the state are from before the step (its first kernel starts behind all of the step before)
  const bool in = c < vdim, fresh = a.positions[b] == 0;
  float* slot = a.state + (int64_t)a.slots[b] * a.slot_stride + (int64_t)h * ((int64_t)dim * vdim + dim + 1);
  float gate = 0.f, w = 0.f;
  if (warp == 0 && in) w = ldf((const E*)a.norm_w + h * vdim + c);
  const float nv = tid < dim && !fresh ? slot[(int64_t)dim * vdim + tid] : 0.f, m0 = fresh ? 0.f : slot[(int64_t)dim * vdim + dim];
  float S[ML_MAXD / 8];
#pragma unroll
  for (int k = 0; k < ML_MAXD / 8; ++k) S[k] = d0 + k < d1 && in && !fresh ? slot[(int64_t)(d0 + k) * vdim + c] : 0.f;
  pdl_wait();
  const float ip = a.gates[(int64_t)b * 2 * a.H + h], fp = a.gates[(int64_t)b * 2 * a.H + a.H + h];
  const float vv0 = in ? ldf((const E*)a.v + (int64_t)b * a.ld + h * vdim + c) : 0.f;
  if (warp == 0 && in) gate = ldf((const E*)a.g + (int64_t)b * a.ld + h * vdim + c);
  float nk = 0.f, nq = 0.f;
  if (tid < dim) {
    nk = ldf((const E*)a.k + (int64_t)b * a.ld + h * dim + tid);
    nq = ldf((const E*)a.q + (int64_t)b * a.ld + h * dim + tid) * a.q_scale;
    ks[tid] = nk; qs[tid] = nq;
  }
  const float it = a.cap * tanhf(ip / a.cap), fc = a.cap * tanhf(fp / a.cap), ft = fminf(fc, 0.f) - log1pf(expf(-fabsf(fc)));
  const float mn = fmaxf(ft + m0, it), fa = expf(ft + m0 - mn), ia = expf(it - mn), vv = ia * vv0;
  __syncthreads();
  float num = 0.f;
#pragma unroll
  for (int k = 0; k < ML_MAXD / 8; ++k)
    if (d0 + k < d1) {
      S[k] = fmaf(fa, S[k], ks[d0 + k] * vv);
      num = fmaf(S[k], qs[d0 + k], num);
      if (in) slot[(int64_t)(d0 + k) * vdim + c] = S[k];
    }
  part[warp][lane] = num;
  const float nn = fmaf(fa, nv, ia * nk), np = warp_sum(tid < dim ? nn * nq : 0.f);
  if (lane == 0) np_s[warp] = np;
  cluster_wait();
  __syncthreads();
  float o = 0.f;
  if (warp == 0) {
    float den = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) { o += part[k][lane]; den += np_s[k]; }
    o = in ? o / (fmaxf(fabsf(den), expf(-mn)) + a.den_eps) : 0.f;
    const float sq = warp_sum(o * o);
    if (lane < (int)gridDim.z)
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_u32((uint32_t)__cvta_generic_to_shared(&squares[blockIdx.z]), (uint32_t)lane)), "f"(sq) : "memory");
  }
  cluster_arrive(); cluster_wait();                            // the squares are there, and all have read n and m
  if (warp == 0 && in) {
    float ss = 0.f;
    for (int k = 0; k < (int)gridDim.z; ++k) ss += squares[k];
    const float inv = a.out_scale / sqrtf(ss / (float)vdim + a.eps);
    stf((E*)a.out + (int64_t)b * a.ldo + h * vdim + c, o * inv * w * (1.f / (1.f + expf(-gate))));
  }
  if (blockIdx.z == 0) {
    if (tid < dim) slot[(int64_t)dim * vdim + tid] = nn;
    if (tid == 0) slot[(int64_t)dim * vdim + dim] = mn;
  }
}

// Decode steps in one launch: at most eight blocks of 32 columns; where heads of few key dimensions fill the SMs many times over, what a
// block costs beside its state weighs more than the launches.  Three launches and one, us, 8 heads of 256 columns: 16 keys 64 requests (4096
// blocks) 31.5 / 33.5, 250 94.7 / 113.6; 32 keys 250 99.8 / 115.3; 64 keys 128 requests 62.3 / 68.1; from 96 keys on ahead everywhere (128
// requests 3 %, of 128 keys 7 %), up to 2048 blocks for all sizes (2 to 60 %).
static bool mlstm_one_launch(const MlstmArgs& a) {
  return a.vdim <= 8 * 32 && (a.dim >= 96 || (int64_t)a.B * a.H * ((a.vdim + 31) / 32) <= 2048);
}
// Clusters of S blocks that run at once on this device: one block an SM, and what is left of a GPC beyond a multiple of S stays empty
// (148, 74, 45, 33, 26, 22, 15 and 15 on a B200).  0: not known.
static int mlstm_clusters(int S) {
  static std::atomic<int> known[16][9];      // [device][S], plus one
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return 0; }
  std::atomic<int>* const at = dev < 16 ? &known[dev][S] : nullptr;
  if (at && at->load(std::memory_order_relaxed)) return at->load(std::memory_order_relaxed) - 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S); cfg.blockDim = dim3(MM_THREADS); cfg.dynamicSmemBytes = sizeof(MlstmTile);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(mlstm_mma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlstmTile)) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, mlstm_mma_kernel<true>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
  if (at) at->store(n + 1, std::memory_order_relaxed);
  return n;
}
// Blocks that share a head's columns of a request (a cluster): as many as leave all clusters running at once, and no more than there are
// chunks.  (48 clusters of three are three more than fit: three prompts of 200 tokens, 4 heads of 16 x 128, 29.4 us with one block,
// 31.8 with three, 24.3 with two.)
static int mlstm_ranks(const MlstmArgs& a) {
  const int64_t blocks = (int64_t)a.B * a.H * ((a.vdim + MM_COLS - 1) / MM_COLS), rows = a.max_rows > 0 ? a.max_rows : a.T - a.B + 1;
  for (int S = (int)std::min<int64_t>(8, (rows + MM_CH - 1) / MM_CH); S > 1; --S)
    if (blocks <= mlstm_clusters(S)) return S;
  return 1;
}
// Tensor-core chunks or the fp32 ones, by estimates (us) from measurements at 8 x 32 x 32 to 4 x 128 x 256 and 1 to 256 requests: a
// tensor-core block fills an SM and takes 9 us beside 7 per 64 tokens of the longest request, an fp32 one shares it with two others,
// 8 us and 1.1 per token (0.6 to 1.1 by head size).  (Blocks that share a head's columns only shorten requests of several chunks, where
// the tensor cores are ahead by far.)  4 x 128 x 256, tensor cores (one block) and fp32: 2 x 1150 tokens 152 / 1278, 200 and 64
// single ones 134 / 290, 8 x 40 36 / 65; 30 x 16 88 / 84, 64 x 8 178 / 73, 60 and 200 single ones 429 / 174, 100 x 2 263 / 60.
static bool mlstm_use_mma(const MlstmArgs& a) {
  const double rows = a.max_rows > 0 ? a.max_rows : a.T - a.B + 1, blocks = (double)a.B * a.H * ((a.vdim + 31) / 32);
  return 9.0 * blocks / 148 + 7.0 * ((int)(rows + 63) / 64) < 8.0 * blocks / (3 * 148) + 1.1 * rows;
}

int mlstm_step(const MlstmArgs& a, cudaStream_t st) {
  if (a.T <= 0 || a.B <= 0) return 0;
  if (a.o_scratch && a.nm_scratch && a.dim <= ML_MAXD && a.dim % 4 == 0 && a.H <= 65535) {
    if (a.T == a.B && mlstm_one_launch(a)) {
      auto kern = a.elt == KGE_ELT_F32 ? mlstm_token_kernel<float> : mlstm_token_kernel<__nv_bfloat16>;
      prefer_max_shared(kern);
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(a.B, a.H, (a.vdim + 31) / 32); cfg.blockDim = dim3(256); cfg.stream = st;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = cfg.gridDim.z;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr; cfg.numAttrs = pdl_for_this_launch() ? 2 : 1;
      KGE_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, a));
      return 0;
    }
    const dim3 grid(a.B, a.H, (a.vdim + ML_COLS - 1) / ML_COLS), g2(a.T + a.B, a.H);
    const int nt = std::min(256, (a.vdim + 31) / 32 * 32);
    KGE_CUDA_OK(launch_pdl(mlstm_log_gates_kernel, dim3((a.T * 2 * a.H + 255) / 256), dim3(256), 0, st, const_cast<float*>(a.gates), a.T, a.H, a.cap));
    const size_t csm_bytes = ((size_t)2 * ML_CH * a.dim + ML_CH * ML_CH + ML_MAXD + 5 * ML_CH + (1 + ML_NSL) * ML_CH * MC_COLS) * 4;
    const dim3 cgrid(a.B, a.H, (a.vdim + MC_COLS - 1) / MC_COLS);
    // tensor-core chunks: bfloat16 rows in 16-byte pieces, key dimensions in steps of 16, at most 256 columns
    const bool mma_ok = a.elt == KGE_ELT_BF16 && a.dim % 16 == 0 && a.vdim % 8 == 0 && a.vdim <= 8 * MM_COLS && a.ld % 8 == 0 &&
                        ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & 15) == 0;
    if (a.T > a.B && mma_ok && mlstm_use_mma(a)) {
      const int Z = (a.vdim + MM_COLS - 1) / MM_COLS, S = mlstm_ranks(a);
      auto kern = S > 1 ? mlstm_mma_kernel<true> : mlstm_mma_kernel<false>;
      KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlstmTile)));
      prefer_max_shared(kern);
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(a.B * S, a.H, Z); cfg.blockDim = dim3(MM_THREADS); cfg.dynamicSmemBytes = sizeof(MlstmTile); cfg.stream = st;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr; cfg.numAttrs = pdl_for_this_launch() ? 2 : 1;
      KGE_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, a));
      if (int rc = mlstm_norm_gate(a, g2, nt, st)) return rc;
      return 0;
    }
    if (a.T > a.B) {
      // some request brings several rows: 32 tokens at a time (single-token requests of the same step are chunks of one)
      static bool smem_set = false;
      if (!smem_set) {
        KGE_CUDA_OK(cudaFuncSetAttribute(mlstm_chunk_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
        KGE_CUDA_OK(cudaFuncSetAttribute(mlstm_chunk_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024));
        smem_set = true;
      }
      if (a.elt == KGE_ELT_F32) KGE_CUDA_OK(launch_pdl(mlstm_chunk_kernel<float>, cgrid, dim3(MC_COLS * ML_NSL), csm_bytes, st, a));
      else KGE_CUDA_OK(launch_pdl(mlstm_chunk_kernel<__nv_bfloat16>, cgrid, dim3(MC_COLS * ML_NSL), csm_bytes, st, a));
      if (a.elt == KGE_ELT_F32) KGE_CUDA_OK(launch_pdl(mlstm_norm_gate_kernel<float>, g2, dim3(nt), 0, st, a));
      else if (int rc = mlstm_norm_gate(a, g2, nt, st)) return rc;
      return 0;
    }
    if (a.elt == KGE_ELT_F32) {
      KGE_CUDA_OK(launch_pdl(mlstm_cols_kernel<float>, grid, dim3(ML_THREADS), 0, st, a));
      KGE_CUDA_OK(launch_pdl(mlstm_norm_gate_kernel<float>, g2, dim3(nt), 0, st, a));
    } else {
      KGE_CUDA_OK(launch_pdl(mlstm_cols_kernel<__nv_bfloat16>, grid, dim3(ML_THREADS), 0, st, a));
      if (int rc = mlstm_norm_gate(a, g2, nt, st)) return rc;
    }
    return 0;
  }
  const int threads = (std::max(a.dim, a.vdim) + 31) / 32 * 32;
  KGE_REQUIRE(threads <= 1024, "mlstm_step: head sizes %d x %d need more than 1024 threads", a.dim, a.vdim);
  const size_t smem = ((size_t)a.dim * a.vdim + 3 * (size_t)a.dim + 64) * 4;
  KGE_REQUIRE(smem <= 227 * 1024, "mlstm_step: a %d x %d state does not fit shared memory", a.dim, a.vdim);
  const dim3 grid(a.B, a.H), block(threads);
  cudaError_t ce;
  if (a.elt == KGE_ELT_F32) {
    cudaFuncSetAttribute(mlstm_step_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    ce = launch_pdl(mlstm_step_kernel<float>, grid, block, smem, st, a);
  } else {
    cudaFuncSetAttribute(mlstm_step_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    ce = launch_pdl(mlstm_step_kernel<__nv_bfloat16>, grid, block, smem, st, a);
  }
  KGE_CUDA_OK(ce);
  return 0;
}

}  // namespace kge
