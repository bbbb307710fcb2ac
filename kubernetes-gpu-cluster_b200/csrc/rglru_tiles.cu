// The gated linear recurrence (RG-LRU) of prompt steps, by tiles of 32 tokens that know nothing of each other, and of decode steps in
// one launch.  S_t = a_t S_(t-1) + b_t is a composition of affine maps: a first kernel forms a_t and b_t of all tokens and each tile's
// composition (A, B); a second one applies the compositions of the tiles before its own (a fma each) and walks its 32 tokens.
// A request's first row starts from the slot's state: its b takes a S_slot in, and its a becomes RESET, which drops what comes from
// the rows before it (another request's, which may be infinite, so no product with zero).
//   rglru_gates_kernel  prompt steps, bfloat16, diagonal blocks of 32, 64, 128 or 160 channels: convolution, both gate projections on tcgen05 and
//                       the coefficients from one read of x; u never leaves shared memory
//   rglru_ab_kernel     prompt steps of any other sizes, and float32: coefficients from gate pre-activations
//   rglru_walk_kernel   the walk behind either, times gelu(y); leaves the new state
//   rglru_step_kernel   decode steps, bfloat16, one row a request: from x to the outputs, products on mma.sync (a block has 16 rows)
// Two prompts of 1156 tokens, width 2560 in 16 blocks, us back to back: convolution 14, gates 2 x 22, coefficients 31, a chain of one
// warp per 32 channels 37 and outputs 15 before, 142 in all; 39 + 17 now, 60 in all (4 x 2048: 383 and 185).  Decode steps of 2, 64 and 200
// requests: 11.6, 29.9 and 37.4 in four launches, 5.3, 16.0 and 32.7 in one.
// What bounds them: the first, issue of the activations and the latency of its stages; the walk, reading a and b (12 bytes a
// number with y) with half of the warps that would fit.
#include <algorithm>

#include "common.cuh"
#include "elt_access.cuh"
#include "f32x2.cuh"
#include "gate_math.cuh"
#include "hybrid_ops.h"

namespace kge {

constexpr int RG_TILE = 32;                    // tokens of a tile
constexpr int RG_MAX_TAPS = 16;

__device__ __forceinline__ bool is_reset(float a) { return __float_as_uint(a) == 0x80000000u; }     // -0: no exponential is
__device__ __forceinline__ float reset_mark() { return -0.f; }
// (A, B) and then (a, b)
__device__ __forceinline__ void rg_compose(float& A, float& B, float a, float b) {
  const bool r = is_reset(a);
  B = r ? b : fmaf(a, B, b);
  A = r ? a : a * A;
}
__device__ __forceinline__ void rg_compose2(f2& A, f2& B, f2 a, f2 b) {
  float A0, A1, B0, B1, a0, a1, b0, b1;
  upk(A, A0, A1); upk(B, B0, B1); upk(a, a0, a1); upk(b, b0, b1);
  rg_compose(A0, B0, a0, b0);
  rg_compose(A1, B1, a1, b1);
  A = pk(A0, A1); B = pk(B0, B1);
}
// a_t and b_t = sqrt(1 - a_t^2) i_t u_t of two numbers from the pre-activations of r and i; rate = -decay * softplus(lam)
__device__ __forceinline__ void rg_coefficients(f2 r, f2 i, f2 u, f2 rate, f2& a, f2& b) {
  const f2 w = mul2(rate, sigmoid2(r));
  a = exp2_(w);
  b = mul2(mul2(complement_root2(w), sigmoid2(i)), u);
}
template <typename E>
__device__ __forceinline__ float rg_rate(const RglruArgs& a, int c) { return -a.decay_c * softplusf_(ldf((const E*)a.lam + c)); }

// V neighbouring channels of a row
template <int V, typename E>
__device__ __forceinline__ f2 rg_load(const E* p) {
  if constexpr (V == 1) return pk(ldf(p), 0.f);
  else if constexpr (sizeof(E) == 4) return *reinterpret_cast<const f2*>(p);
  else { const uint32_t w = *reinterpret_cast<const uint32_t*>(p); return pk(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
}
template <int V, typename E>
__device__ __forceinline__ void rg_store(E* p, f2 v) {
  float x, y;
  upk(v, x, y);
  if constexpr (V == 1) stf(p, x);
  else if constexpr (sizeof(E) == 4) *reinterpret_cast<f2*>(p) = v;
  else { const __nv_bfloat162 h = __floats2bfloat162_rn(x, y); *reinterpret_cast<uint32_t*>(p) = *reinterpret_cast<const uint32_t*>(&h); }
}

// the slots' numbers start anywhere
template <int V>
__device__ __forceinline__ f2 rg_state(const float* p) { return pk(p[0], V == 2 ? p[V - 1] : 0.f); }
template <int V>
__device__ __forceinline__ void rg_keep(float* p, f2 v) {
  float x, y;
  upk(v, x, y);
  p[0] = x;
  if (V == 2) p[V - 1] = y;
}

// One tile and 32 x V channels per block, V channels a thread and eight of the tile's rows a warp, all asked for at once; the warps' compositions
// meet in shared memory.  With the 32 rows in one thread, four at a time, 40 tokens of 1536
// channels waited for eight trips to memory one after another: 22 us, 5.7 now; 600 tokens 23 and 9.4.
constexpr int RB_ROWS = 8, RB_WARPS = RG_TILE / RB_ROWS;
template <typename E, int V>
__global__ void __launch_bounds__(RB_WARPS * 32) rglru_ab_kernel(RglruArgs a, float* gates) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ f2 parts[RB_WARPS - 1][2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = (blockIdx.y * 32 + lane) * V, t0 = blockIdx.x * RG_TILE + warp * RB_ROWS, n = min(RB_ROWS, a.T - t0);
  const bool in = c < a.width;
  const int at = in ? c : 0;
  f2 gr[RB_ROWS], gi[RB_ROWS], uv[RB_ROWS];
  // (a warp's own rows, the last of them again where there are fewer: loads under conditions came one by one)
  if (n > 0) {
#pragma unroll
    for (int k = 0; k < RB_ROWS; ++k) {
      const int t = t0 + min(k, n - 1);
      const float* gt = gates + (int64_t)t * 2 * a.width + at;
      gr[k] = rg_load<V>(gt); gi[k] = rg_load<V>(gt + a.width);
      uv[k] = rg_load<V>((const E*)a.u + (int64_t)t * a.width + at);
    }
  }
  // lane k knows row k: whether it is its request's first, and where a state before it lies
  bool first = false, old = false;
  int64_t slot = 0;
  if (lane < n && lane < RB_ROWS) {
    const int t = t0 + lane, b = a.token_req[t];
    first = a.qsl[b] == t;
    old = first && a.positions[t] > 0;
    slot = (int64_t)a.slots[b] * a.slot_stride;
  }
  const uint32_t firsts = __ballot_sync(0xffffffffu, first), olds = __ballot_sync(0xffffffffu, old);
  const f2 rate = in ? pk(rg_rate<E>(a, c), V == 2 ? rg_rate<E>(a, c + V - 1) : 0.f) : pk1(0.f);
  f2 s0[RB_ROWS], A = pk1(1.f), B = pk1(0.f);
#pragma unroll
  for (int k = 0; k < RB_ROWS; ++k) {
    const int64_t from = __shfl_sync(0xffffffffu, slot, k);
    s0[k] = in && (olds >> k & 1) ? rg_state<V>(a.state + from + c) : pk1(0.f);
  }
#pragma unroll
  for (int k = 0; k < RB_ROWS; ++k) {
    if (!in || k >= n) break;
    f2 av, bv;
    rg_coefficients(gr[k], gi[k], uv[k], rate, av, bv);
    if (firsts >> k & 1) {
      bv = fma2(av, s0[k], bv);
      av = pk1(reset_mark());
    }
    float* gt = gates + (int64_t)(t0 + k) * 2 * a.width + c;
    rg_store<V>(gt, av);
    rg_store<V>(gt + a.width, bv);
    rg_compose2(A, B, av, bv);
  }
  if (warp > 0) { parts[warp - 1][0][lane] = A; parts[warp - 1][1][lane] = B; }
  __syncthreads();
  if (warp > 0 || !in) return;
#pragma unroll
  for (int w = 0; w < RB_WARPS - 1; ++w) rg_compose2(A, B, parts[w][0][lane], parts[w][1][lane]);      // (1, 0) behind the last row
  float* to = a.tiles + (int64_t)blockIdx.x * 2 * a.width + c;
  rg_store<V>(to, A);
  rg_store<V>(to + a.width, B);
}

// The walk: PART of a tile's rows are in flight at a time, the first ones before anything else.  Eight leave room for twelve blocks an SM; sixteen
// halve the trips to memory of launches that leave SMs idle (40 tokens of 1536 channels 9.5 us and 7.6, 600 12.0 and
// 11.3).  Blocks behind the tiles, one a request, bring the
// convolution's inputs up to date (in the walk it cost steps with many requests a trip to memory a row).
template <typename E, int V, int PART>
__global__ void __launch_bounds__(64, PART == 8 ? 12 : 6) rglru_walk_kernel(RglruArgs a, const float* __restrict__ gates, int tiles) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ int slot_s[RG_TILE], starts_s;                    // of each row; the row at which the first row's request begins
  __shared__ uint32_t ends_s;                                  // the rows that are their request's last
  const int c = (blockIdx.y * 64 + threadIdx.x) * V;
  const bool in = c < a.width;
  const int64_t ld = 2 * (int64_t)a.width;
  if ((int)blockIdx.x >= tiles) {
    const int b = blockIdx.x - tiles, rs = a.qsl[b], len = a.qsl[b + 1] - rs;
    if (len <= 0 || !in) return;
    const int p0 = a.positions[rs];
    float* tail = a.state + (int64_t)a.slots[b] * a.slot_stride + a.width + c;
    // what is read of the old inputs lies behind what is written
    auto next = [&](int j) -> f2 {
      const int back = a.taps - 1 - j, sp = p0 + len - back;
      if (back <= len) return rg_load<V>((const E*)a.yx + (int64_t)(rs + len - back) * ld + a.width + c);
      return sp >= 0 ? rg_state<V>(tail + (int64_t)(len + j) * a.width) : pk1(0.f);
    };
    constexpr int J = 3;                                       // at once, as four taps want
    for (int j0 = 0; j0 < a.taps - 1; j0 += J) {
      f2 v[J];
#pragma unroll
      for (int j = 0; j < J; ++j) if (j0 + j < a.taps - 1) v[j] = next(j0 + j);
#pragma unroll
      for (int j = 0; j < J; ++j) if (j0 + j < a.taps - 1) rg_keep<V>(tail + (int64_t)(j0 + j) * a.width, v[j]);
    }
    return;
  }
  // addresses as a row's, the same for all threads, and a 32-bit column
  const int tile = blockIdx.x, t0 = tile * RG_TILE, n = min(RG_TILE, a.T - t0);
  const uint32_t cu = (uint32_t)c;
  f2 av[PART], bv[PART], yv[PART];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int k = 0; k < PART; ++k) {
      const int64_t r = (int64_t)(t0 + min(k0 + k, n - 1)) * ld;
      av[k] = rg_load<V>(gates + r + cu);
      bv[k] = rg_load<V>(gates + r + a.width + cu);
      yv[k] = rg_load<V>((const E*)a.yx + r + cu);
    }
  };
  if (in) fetch(0);
  if (threadIdx.x < RG_TILE) {
    const int t = t0 + min((int)threadIdx.x, n - 1), b = a.token_req[t];
    const uint32_t ends = __ballot_sync(0xffffffffu, (int)threadIdx.x < n && (t + 1 == a.T || a.token_req[min(t + 1, a.T - 1)] != b));
    slot_s[threadIdx.x] = a.slots[b];
    if (threadIdx.x == 0) { ends_s = ends; starts_s = a.qsl[b]; }
  }
  __syncthreads();
  if (!in) return;
  const uint32_t ends = ends_s;
  // what the request's earlier tiles make of its state: none of it where the tile's first row is the request's
  f2 S = pk1(0.f);
  if (starts_s < t0) {
    constexpr int G = 4;
    for (int s0 = starts_s / RG_TILE; s0 < tile; s0 += G) {
      f2 A[G], B[G];
#pragma unroll
      for (int k = 0; k < G; ++k) {
        const float* from = a.tiles + (int64_t)min(s0 + k, tile - 1) * ld;
        A[k] = rg_load<V>(from + cu);
        B[k] = rg_load<V>(from + a.width + cu);
      }
#pragma unroll
      for (int k = 0; k < G; ++k)
        if (s0 + k < tile) {
          f2 none = pk1(0.f);
          rg_compose2(none, S, A[k], B[k]);
        }
    }
  }
  const bool whole = n == RG_TILE && starts_s < t0 && (ends & 0x7fffffffu) == 0;      // no request begins in the tile
#pragma unroll 1
  for (int k0 = 0; k0 < n; k0 += PART) {
    E* out = (E*)a.out + (int64_t)(t0 + k0) * a.width;
    if (whole) {
#pragma unroll
      for (int k = 0; k < PART; ++k) {
        S = fma2(av[k], S, bv[k]);
        rg_store<V>(out + (int64_t)k * a.width + cu, mul2(S, gelu_tanh2(yv[k])));
      }
      if (k0 + PART == RG_TILE && ends) rg_keep<V>(a.state + (int64_t)slot_s[RG_TILE - 1] * a.slot_stride + c, S);
    } else {
#pragma unroll
      for (int k = 0; k < PART; ++k) {
        f2 none = pk1(0.f);
        rg_compose2(none, S, av[k], bv[k]);
        if (k0 + k < n) rg_store<V>(out + (int64_t)k * a.width + cu, mul2(S, gelu_tanh2(yv[k])));
        if (ends >> (k0 + k) & 1) rg_keep<V>(a.state + (int64_t)slot_s[k0 + k] * a.slot_stride + c, S);
      }
    }
    if (k0 + PART < n) fetch(k0 + PART);
  }
}

// The gate products of decode steps, on mma.sync: a block has 16 rows and `cols` columns of one diagonal block, the weights of both gates in
// shared memory; a warp has eight columns of both gates, so r and i of a number meet in one thread.
__device__ __forceinline__ void rg_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void rg_ldsm(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
// acc[gate] = 16 rows of U x the warp's eight columns of W [gate][cols][bw]
__device__ __forceinline__ void rg_products(float (&acc)[2][4], const __nv_bfloat16* W, const __nv_bfloat16* U, int cols, int n0, int bw, int lane) {
  const int ldw = bw + 8;                                      // rows 16 bytes apart in their banks
#pragma unroll
  for (int q = 0; q < 2; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.f;
  const __nv_bfloat16* w = W + (int64_t)((lane >> 4) * cols + n0 + (lane & 7)) * ldw + ((lane >> 3) & 1) * 8;
  const __nv_bfloat16* u = U + (lane & 15) * ldw + (lane >> 4) * 8;
#pragma unroll 2
  for (int k = 0; k < bw; k += 16) {
    uint32_t bf[4], af[4];                                     // r's two halves of 16 keys, i's
    rg_ldsm(bf, w + k);
    rg_ldsm(af, u + k);
    rg_mma(acc[0], af, bf[0], bf[1]);
    rg_mma(acc[1], af, bf[2], bf[3]);
  }
}
__device__ __forceinline__ void rg_fetch_weights(__nv_bfloat16* W, const RglruArgs& a, int z, int c0, int cols, int bw) {
  const int pieces = bw / 8;
  for (int r = threadIdx.x >> 5; r < 2 * cols; r += blockDim.x >> 5) {
    const __nv_bfloat16* src = (const __nv_bfloat16*)(r >= cols ? a.w_i : a.w_r) + ((int64_t)z * bw + c0 + r - (r >= cols ? cols : 0)) * bw;
    for (int p = threadIdx.x & 31; p < pieces; p += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(W + (int64_t)r * (bw + 8) + p * 8)), "l"(src + p * 8) : "memory");
  }
}

struct RgRow { int back, pos; const float* slot; };           // rows of the step before it that are its request's; position; state
__device__ __forceinline__ RgRow rg_row(const RglruArgs& a, int t) {
  const int b = a.token_req[t];
  return RgRow{t - a.qsl[b], a.positions[t], a.state + (int64_t)a.slots[b] * a.slot_stride};
}

// Weights and bias of the convolution's eight channels from c on.  TAPS 4: a channel's taps lie side by side, 64 bytes for eight; 0: any.
template <int TAPS>
struct RgTaps {
  uint4 q[TAPS ? TAPS : 1];
  const __nv_bfloat16* w;
  int taps;
  __device__ __forceinline__ RgTaps(const RglruArgs& a, int c) : w((const __nv_bfloat16*)a.conv_w + (int64_t)c * (TAPS ? TAPS : a.taps)), taps(TAPS ? TAPS : a.taps) {
#pragma unroll
    for (int i = 0; i < TAPS; ++i) q[i] = *reinterpret_cast<const uint4*>(w + i * 8);
  }
  __device__ __forceinline__ float get(int e, int j) const {
    if constexpr (TAPS > 0) {
      const uint4& v = q[(e * TAPS + j) / 8];
      const int at = (e * TAPS + j) % 8;
      const uint32_t two = at < 2 ? v.x : at < 4 ? v.y : at < 6 ? v.z : v.w;
      return (at & 1) ? bf_hi(two) : bf_lo(two);
    } else {
      return ldf(w + (int64_t)e * taps + j);
    }
  }
  __device__ __forceinline__ f2 pair(int e, int j) const { return pk(get(e, j), get(e + 1, j)); }
};
__device__ __forceinline__ void rg_wide(uint4 q, f2 (&v)[4]) {
  v[0] = pk(bf_lo(q.x), bf_hi(q.x)); v[1] = pk(bf_lo(q.y), bf_hi(q.y)); v[2] = pk(bf_lo(q.z), bf_hi(q.z)); v[3] = pk(bf_lo(q.w), bf_hi(q.w));
}
__device__ __forceinline__ uint32_t rg_narrow(f2 v) { float x, y; upk(v, x, y); return pack_bf2(x, y); }

// u of eight channels from c on of row t, any row: inputs before the step are the slot's last taps - 1 ones, zeros before position 0
template <int TAPS>
__device__ __forceinline__ void rg_conv_any(f2 (&acc)[4], const RglruArgs& a, const RgTaps<TAPS>& w, const RgRow& m, int t, int c) {
  const __nv_bfloat16* x = (const __nv_bfloat16*)a.yx + (int64_t)t * 2 * a.width + a.width + c;
  const int taps = TAPS ? TAPS : w.taps;
#pragma unroll(TAPS ? TAPS : 1)
  for (int j = 0; j < taps; ++j) {
    const int back = taps - 1 - j;
    f2 v[4];
    if (back <= m.back) {
      rg_wide(*reinterpret_cast<const uint4*>(x - (int64_t)back * 2 * a.width), v);
    } else {
      const float* tail = m.slot + a.width + (int64_t)(m.back - back + taps - 1) * a.width + c;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = back <= m.pos ? pk(tail[2 * e], tail[2 * e + 1]) : pk1(0.f);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = fma2(w.pair(2 * e, j), v[e], acc[e]);
  }
}

// Prompt steps.  The products are tcgen05 MMAs with the weights as their 128 rows: a TMEM lane is a channel and the columns are tokens, so
// that a thread has a channel's r and i of 32 tokens in a row, composes them by itself, and a warp stores whole lines.  (On mma.sync,
// which takes 32 cycles a quarter of an SM for 16 x 8 x 16 numbers, the products alone took 26 us of 60 at 2312 x 2560.)
// One block an SM keeps its diagonal block's weights (swizzled by 64 bytes: any multiple of 32 channels without padding) and walks over
// a share of the tokens with two groups of warps, each on tiles of 64 of its own, so that one's products and loads are behind the
// other's arithmetic.  32 channels are a quadrant of lanes: what is left of a diagonal block beyond 128 channels is repeated in all
// quadrants of a second tile of rows, of which the warps take one half of the tokens each.
constexpr int RT_N = 64;                       // tokens of a tile
constexpr uint32_t RT_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(RT_N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
__device__ __forceinline__ uint64_t rt_desc(uint32_t saddr) {  // K-major rows of 64 bytes, atoms of 8 rows 512 bytes apart, SWIZZLE_64B
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
__device__ __forceinline__ void rt_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a), "l"(b), "r"(RT_IDESC), "r"(acc) : "memory");
}
__device__ __forceinline__ void rt_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
__host__ __device__ constexpr int rt_row_tiles(int quads) { return (quads + 3) / 4; }                  // quads: groups of 32 channels
// the 32 channels in quadrant q of row tile m: in full tiles one after another, the rest (one group or two) in turn
__host__ __device__ constexpr int rt_channels(int quads, int m, int q) { return 4 * m + (4 * m + 4 <= quads ? q : quads - 4 * m == 2 ? q & 1 : 0); }
__host__ __device__ constexpr bool rt_fits(int bw) { return bw == 32 || bw == 64 || bw == 128 || bw == 160; }

template <int QUADS, int TAPS>
__global__ void __launch_bounds__(QUADS * 128) rglru_gates_kernel(RglruArgs a, float* gates, int units) {
  typedef __nv_bfloat16 E;
  constexpr int BW = QUADS * 32, MT = rt_row_tiles(QUADS), PIECES = BW / 8, GROUP = QUADS * 64, ROWS_A = QUADS * 128 * 64, ROWS_U = RT_N * 64;
  constexpr uint32_t COLS = 2 * MT * RT_N;                     // of a group: [gate][row tile][token]
  extern __shared__ __align__(1024) unsigned char rg_raw[];
  // no static shared memory: the dynamic window starts where the swizzle's pattern does
  uint64_t* bars = reinterpret_cast<uint64_t*>(rg_raw + 2 * MT * ROWS_A + 2 * QUADS * ROWS_U);
  uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 2);
  const uint32_t sA = (uint32_t)__cvta_generic_to_shared(rg_raw);                                      // [gate][row tile][k / 32][128 rows][64 bytes]
  if (sA & 511u) __trap();
  const int tid = threadIdx.x, lane = tid & 31, warp = uniform_warp(), grp = warp >= QUADS * 2, gw = warp - grp * QUADS * 2, gt = tid - grp * GROUP, quad = warp & 3;
  const uint32_t offU = 2 * MT * ROWS_A + grp * QUADS * ROWS_U;                                         // [k / 32][64 tokens][64 bytes]
  const int z = blockIdx.y, taps = TAPS ? TAPS : a.taps;
  const int64_t ld = 2 * (int64_t)a.width;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&tmem_slot)), "n"(2 * COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    if (lane < 2) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(&bars[lane])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < 2 * MT * 128 * PIECES; i += QUADS * 128) {
    const int r = i / PIECES, c = i - r * PIECES, row = r & 127, m = r / 128 % MT, gate = r / (128 * MT);
    const E* src = (const E*)(gate ? a.w_i : a.w_r) + ((int64_t)z * BW + rt_channels(QUADS, m, row >> 5) * 32 + (row & 31)) * BW + c * 8;
    const uint32_t dst = sA + (gate * MT + m) * ROWS_A + (c >> 2) * (128 * 64) + row * 64 + (((c & 3) ^ (row >> 1 & 3)) << 4);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  }
  // this warp's unit of a tile: 32 channels, half of the tokens
  const int m = gw < QUADS / 4 * 8 ? gw / 8 : MT - 1, rest = QUADS - 4 * m;
  const int half = rest >= 4 ? gw / 4 & 1 : rest == 2 ? quad >> 1 : gw & 1, ch32 = rt_channels(QUADS, m, quad), ch = z * BW + ch32 * 32 + lane;
  const f2 rate = pk1(rg_rate<E>(a, ch)), br = pk1(a.b_r ? ldf((const E*)a.b_r + ch) : 0.f), bi = pk1(a.b_i ? ldf((const E*)a.b_i + ch) : 0.f);
  pdl_wait();
  asm volatile("cp.async.wait_all;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // the columns are held: blocks of a later kernel that took them first would wait for this one
  pdl_launch_dependents();
  const uint32_t tmem = tmem_slot + grp * COLS, bar = (uint32_t)__cvta_generic_to_shared(&bars[grp]);
  // the block's share of the units of 32 tokens, and what of it ends at the last token
  const int u0 = (int)((int64_t)units * blockIdx.x / gridDim.x), u1 = (int)((int64_t)units * (blockIdx.x + 1) / gridDim.x), end = min(u1 * RG_TILE, a.T);
  const int q4 = gt / PIECES * 4, p = gt % PIECES, cc = z * BW + p * 8;                                 // this thread's four rows and eight channels of the convolution
  const RgTaps<TAPS> w(a, cc);
  uint32_t parity = 0;
#pragma unroll 1
  for (int t0 = u0 * RG_TILE + grp * RT_N; t0 < end; t0 += 2 * RT_N, parity ^= 1) {
    const int tq = t0 + q4;
    {
      // u of the tile; where the four rows and their inputs are one request's rows of this step, seven loads are all there is
      f2 acc[4][4];
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[0][e] = acc[1][e] = acc[2][e] = acc[3][e] = rg_load<2>((const E*)a.conv_b + cc + 2 * e);
      const bool all = TAPS > 0 && tq >= TAPS - 1 && tq + 4 <= end && a.token_req[max(tq - (TAPS - 1), 0)] == a.token_req[min(tq + 3, a.T - 1)];
      const E* x = (const E*)a.yx + (int64_t)tq * ld + a.width + cc;
      if (all) {
        uint4 xr[TAPS + 3];
#pragma unroll
        for (int s = 0; s < TAPS + 3; ++s) xr[s] = *reinterpret_cast<const uint4*>(x + (s - (TAPS - 1)) * ld);
#pragma unroll
        for (int s = 0; s < TAPS + 3; ++s) {
          f2 v[4];
          rg_wide(xr[s], v);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (s - k >= 0 && s - k < TAPS)
#pragma unroll
              for (int e = 0; e < 4; ++e) acc[k][e] = fma2(w.pair(2 * e, s - k), v[e], acc[k][e]);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (tq + k < end) rg_conv_any(acc[k], a, w, rg_row(a, tq + k), tq + k, cc);
      }
      // the group has read the tile before
      asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(GROUP) : "memory");
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int r = q4 + k;
        *reinterpret_cast<uint4*>(rg_raw + offU + (p >> 2) * ROWS_U + r * 64 + (((p & 3) ^ (r >> 1 & 3)) << 4)) =
            make_uint4(rg_narrow(acc[k][0]), rg_narrow(acc[k][1]), rg_narrow(acc[k][2]), rg_narrow(acc[k][3]));
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(GROUP) : "memory");
    if (gw == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint64_t bd = rt_desc(sA + offU);
#pragma unroll 1
        for (int g = 0; g < 2 * MT; ++g) {
          const uint64_t ad = rt_desc(sA + g * ROWS_A);
#pragma unroll
          for (int k = 0; k < 2 * QUADS; ++k)
            rt_mma(tmem + g * RT_N, ad + (uint64_t)(((k >> 1) * (128 * 64) + (k & 1) * 32) >> 4), bd + (uint64_t)(((k >> 1) * ROWS_U + (k & 1) * 32) >> 4), k > 0);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
      }
      __syncwarp();
    }
    const int tu = t0 + half * RG_TILE, n = min(end - tu, RG_TILE);
    // one request's rows, none of them its first: its earlier row is the one before the tile
    const bool inner = n == RG_TILE && tu > 0 && a.token_req[max(tu - 1, 0)] == a.token_req[tu + max(n, 1) - 1];
    mbar_wait(bar, parity);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (n > 0) {
      float A = 1.f, B = 0.f;
      float* to = gates + tu * ld + ch;
#pragma unroll 1
      for (int c0 = 0; c0 < RG_TILE; c0 += 16) {
        uint32_t rr[16], ri[16];
        const uint32_t at = tmem + (uint32_t)(quad << 21) + m * RT_N + half * RG_TILE + c0;
        rt_ld16(at, rr);
        rt_ld16(at + MT * RT_N, ri);
        tmem_wait_ld(rr, ri);
        const unsigned char* us = rg_raw + offU + ch32 * ROWS_U + (half * RG_TILE + c0) * 64 + (lane & 7) * 2;
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          const unsigned char* uk = us + k * 64 + (((lane >> 3) ^ (k >> 1 & 3)) << 4);
          const f2 u = pk(ldf(reinterpret_cast<const E*>(uk)), ldf(reinterpret_cast<const E*>(uk + 64)));
          f2 av, bv;
          rg_coefficients(add2(pk(__uint_as_float(rr[k]), __uint_as_float(rr[k + 1])), br), add2(pk(__uint_as_float(ri[k]), __uint_as_float(ri[k + 1])), bi), u, rate, av, bv);
          float a2[2], b2[2];
          upk(av, a2[0], a2[1]);
          upk(bv, b2[0], b2[1]);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            if (!inner) {
              const int t = tu + c0 + k + j;
              if (t >= end) break;
              const RgRow r = rg_row(a, t);
              if (r.back == 0) {
                if (r.pos > 0) b2[j] = fmaf(a2[j], r.slot[ch], b2[j]);
                a2[j] = reset_mark();
              }
              rg_compose(A, B, a2[j], b2[j]);
            } else {
              B = fmaf(a2[j], B, b2[j]);
              A *= a2[j];
            }
            to[0] = a2[j];
            to[a.width] = b2[j];
            to += ld;
          }
        }
      }
      float* tt = a.tiles + (tu / RG_TILE) * ld + ch;
      tt[0] = A;
      tt[a.width] = B;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "n"(2 * COLS) : "memory");
}

// Decode steps: 16 requests of one row each per block, from x to the outputs.  The blocks of a diagonal block form a cluster: all read
// the convolution's old inputs of all its channels, and each brings its own columns' up to date when the others have read them.
template <int TAPS>
__global__ void __launch_bounds__(320) rglru_step_kernel(RglruArgs a, int bw, int cols) {
  pdl_launch_dependents();
  typedef __nv_bfloat16 E;
  extern __shared__ __align__(16) unsigned char rg_raw[];
  const int ldw = bw + 8;
  E* W = reinterpret_cast<E*>(rg_raw);
  E* U = W + 2 * cols * ldw;                                   // [16][bw]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, t0 = blockIdx.x * 16, n = min(16, a.T - t0);
  const int z = blockIdx.y, c0 = blockIdx.z * cols, n0 = warp * 8, pieces = bw / 8, taps = TAPS ? TAPS : a.taps;
  rg_fetch_weights(W, a, z, c0, cols, bw);
  const int ch = z * bw + c0 + n0 + 2 * t4;
  const f2 rate = pk(rg_rate<E>(a, ch), rg_rate<E>(a, ch + 1));
  const f2 br = a.b_r ? rg_load<2>((const E*)a.b_r + ch) : pk1(0.f), bi = a.b_i ? rg_load<2>((const E*)a.b_i + ch) : pk1(0.f);
  // slots, positions and the state are from before the step (its first kernel starts behind all of the step before)
  auto row_of = [&](int t) { return RgRow{0, a.positions[t], a.state + (int64_t)a.slots[t] * a.slot_stride}; };
  float* slot[2];
  f2 S[2], y[2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (g + 8 * h < n) {
      const RgRow r = row_of(t0 + g + 8 * h);
      slot[h] = const_cast<float*>(r.slot);
      S[h] = r.pos > 0 ? rg_state<2>(r.slot + ch) : pk1(0.f);
    }
  pdl_wait();
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (g + 8 * h < n) y[h] = rg_load<2>((const E*)a.yx + (int64_t)(t0 + g + 8 * h) * 2 * a.width + ch);
  for (int i = tid; i < 16 * pieces; i += blockDim.x) {
    const int r = i / pieces, p = (i - r * pieces) * 8, c = z * bw + p;
    f2 acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = r < n ? rg_load<2>((const E*)a.conv_b + c + 2 * e) : pk1(0.f);
    if (r < n) rg_conv_any(acc, a, RgTaps<TAPS>(a, c), row_of(t0 + r), t0 + r, c);
    *reinterpret_cast<uint4*>(U + r * ldw + p) = make_uint4(rg_narrow(acc[0]), rg_narrow(acc[1]), rg_narrow(acc[2]), rg_narrow(acc[3]));
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  cluster_arrive();                                            // the old inputs have been read
  float acc[2][4];
  rg_products(acc, W, U, cols, n0, bw, lane);
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (g + 8 * h < n) {
      const uint32_t uu = *reinterpret_cast<const uint32_t*>(U + (g + 8 * h) * ldw + c0 + n0 + 2 * t4);
      f2 av, bv;
      rg_coefficients(add2(pk(acc[0][2 * h], acc[0][2 * h + 1]), br), add2(pk(acc[1][2 * h], acc[1][2 * h + 1]), bi), pk(bf_lo(uu), bf_hi(uu)), rate, av, bv);
      const f2 s = fma2(av, S[h], bv);
      rg_keep<2>(slot[h] + ch, s);
      rg_store<2>((E*)a.out + (int64_t)(t0 + g + 8 * h) * a.width + ch, mul2(s, gelu_tanh2(y[h])));
    }
  cluster_wait();
  for (int i = tid; i < n * cols; i += blockDim.x) {
    const int r = i / cols, c = z * bw + c0 + i - r * cols, t = t0 + r;
    const RgRow m = row_of(t);
    float* tail = const_cast<float*>(m.slot) + a.width + c;
    const float x = ldf((const E*)a.yx + (int64_t)t * 2 * a.width + a.width + c);
    auto next = [&](int j) { return j == taps - 2 ? x : m.pos + 1 - (taps - 1) + j >= 0 ? tail[(int64_t)(j + 1) * a.width] : 0.f; };
    if constexpr (TAPS > 1) {
      float v[TAPS - 1];
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) v[j] = next(j);
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) tail[(int64_t)j * a.width] = v[j];
    } else {
      for (int j = 0; j < taps - 1; ++j) tail[(int64_t)j * a.width] = next(j);
    }
  }
}

static bool rg_rows_ok(const RglruArgs& a) {
  return a.elt == KGE_ELT_BF16 && a.blocks > 0 && a.blocks <= 65535 && a.width % a.blocks == 0 && a.taps >= 1 && a.taps <= RG_MAX_TAPS &&
         ((reinterpret_cast<uintptr_t>(a.yx) | reinterpret_cast<uintptr_t>(a.w_r) | reinterpret_cast<uintptr_t>(a.w_i) | reinterpret_cast<uintptr_t>(a.conv_b) | reinterpret_cast<uintptr_t>(a.out)) & 15) == 0 &&
         ((reinterpret_cast<uintptr_t>(a.b_r) | reinterpret_cast<uintptr_t>(a.b_i)) & 3) == 0;
}
bool rglru_step_ok(const RglruArgs& a) { return rg_rows_ok(a) && rglru_step_warps(a.width / a.blocks) > 0; }
bool rglru_gates_ok(const RglruArgs& a) { return rg_rows_ok(a) && rt_fits(a.width / a.blocks); }

static bool rg_four_taps(const RglruArgs& a) { return a.taps == 4 && (reinterpret_cast<uintptr_t>(a.conv_w) & 15) == 0; }

template <int TAPS>
static int rg_step(const RglruArgs& a, cudaStream_t st) {
  const int bw = a.width / a.blocks, groups = rglru_step_warps(bw), cols = groups * 8, parts = bw / cols;
  auto kern = rglru_step_kernel<TAPS>;
  KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (2 * 80 + 16) * (256 + 8) * 2));
  prefer_max_shared(kern);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.T + 15) / 16, a.blocks, parts); cfg.blockDim = dim3(32 * groups); cfg.dynamicSmemBytes = (size_t)(2 * cols + 16) * (bw + 8) * 2; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = parts;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl_for_this_launch() ? 2 : 1;
  KGE_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, a, bw, cols));
  return 0;
}

template <int QUADS, int TAPS>
static int rg_gates(const RglruArgs& a, cudaStream_t st) {
  constexpr size_t smem = (size_t)2 * rt_row_tiles(QUADS) * QUADS * 128 * 64 + 2 * QUADS * RT_N * 64 + 32;
  auto kern = rglru_gates_kernel<QUADS, TAPS>;
  KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int units = (a.T + RG_TILE - 1) / RG_TILE;
  KGE_CUDA_OK(launch_pdl(kern, dim3(std::min(units, std::max(1, 148 / a.blocks)), a.blocks), dim3(QUADS * 128), smem, st, a, const_cast<float*>(a.gates), units));
  return 0;
}
template <int QUADS>
static int rg_gates(const RglruArgs& a, cudaStream_t st) { return rg_four_taps(a) ? rg_gates<QUADS, 4>(a, st) : rg_gates<QUADS, 0>(a, st); }

int rglru_step(const RglruArgs& a, cudaStream_t st) {
  KGE_REQUIRE(rglru_step_ok(a) && a.T == a.B, "rglru_step: %d rows of %d requests, width %d", a.T, a.B, a.width);
  return a.T <= 0 ? 0 : rg_four_taps(a) ? rg_step<4>(a, st) : rg_step<0>(a, st);
}

int rglru_gates(const RglruArgs& a, cudaStream_t st) {
  KGE_REQUIRE(rglru_gates_ok(a) && a.tiles, "rglru_gates: width %d in %d blocks", a.width, a.blocks);
  if (a.T <= 0) return 0;
  switch (a.width / a.blocks) {
    case 32: return rg_gates<1>(a, st);
    case 64: return rg_gates<2>(a, st);
    case 128: return rg_gates<4>(a, st);
    default: return rg_gates<5>(a, st);
  }
}

// Two channels a thread where the rows allow it.
static bool rg_pairs(const RglruArgs& a) {
  return a.width % 2 == 0 && ((reinterpret_cast<uintptr_t>(a.gates) | reinterpret_cast<uintptr_t>(a.yx) | reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.u) | reinterpret_cast<uintptr_t>(a.tiles)) & 7) == 0;
}

template <typename E, int V>
static int rg_by_channel(const RglruArgs& a, bool walk, cudaStream_t st) {
  const dim3 grid((a.T + RG_TILE - 1) / RG_TILE, (a.width + 32 * V - 1) / (32 * V));
  KGE_REQUIRE(grid.y <= 65535 && a.tiles, "rglru: width %d", a.width);
  const dim3 wgrid(grid.x + a.B, (a.width + 64 * V - 1) / (64 * V));
  auto walker = V == 2 && (int64_t)wgrid.x * wgrid.y <= 6 * 148 ? rglru_walk_kernel<E, V, V == 2 ? 16 : 8> : rglru_walk_kernel<E, V, 8>;
  if (walk) KGE_CUDA_OK(launch_pdl(walker, wgrid, dim3(64), 0, st, a, a.gates, (int)grid.x));
  else KGE_CUDA_OK(launch_pdl(rglru_ab_kernel<E, V>, grid, dim3(RB_WARPS * 32), 0, st, a, const_cast<float*>(a.gates)));
  return 0;
}

static int rg_by_channel(const RglruArgs& a, bool walk, cudaStream_t st) {
  if (a.T <= 0) return 0;
  KGE_REQUIRE(a.taps >= 1 && a.taps <= RG_MAX_TAPS, "rglru: %d taps (1..%d)", a.taps, RG_MAX_TAPS);
  if (a.elt == KGE_ELT_F32) return rg_pairs(a) ? rg_by_channel<float, 2>(a, walk, st) : rg_by_channel<float, 1>(a, walk, st);
  return rg_pairs(a) ? rg_by_channel<__nv_bfloat16, 2>(a, walk, st) : rg_by_channel<__nv_bfloat16, 1>(a, walk, st);
}
int rglru_coefficients(const RglruArgs& a, cudaStream_t st) { return rg_by_channel(a, false, st); }
int rglru_walk(const RglruArgs& a, cudaStream_t st) { return rg_by_channel(a, true, st); }

}  // namespace kge
