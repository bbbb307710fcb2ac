// Paged attention with a linear distance bias per head, a chunk mask, an optional soft cap of the scores and an optional
// sink logit per head in the softmax denominator, for any key / value head size, in bfloat16 or float32 storage.  One warp per (query row, head): 32 keys at a time, one key per lane for the scores (q in shared
// memory), softmax statistics in fp32 across the warp, then the lanes split the value columns.  Only keys of the
// query's own chunk are read, so the cost per query is bounded by the chunk size whatever the context length.
#include <algorithm>

#include "common.cuh"
#include "elt_access.cuh"
#include "hybrid_ops.h"

namespace kge {

constexpr int ATT_WARPS = 4, ATT_MAXV = 32;   // value columns per lane at most: vdim <= 32 * ATT_MAXV

// Keys of a row with a window: first the `prefix` keys - kept first tokens that have left the window (their own rows of
// the caches) or pooled blocks that lie wholly before it (rows of the pooled caches) - then the window's tokens.
__device__ __forceinline__ int prefix_keys(const AttnBiasArgs& a, int i) {
  if (a.window <= 0 || i < a.window) return 0;
  const int before = i - a.window + 1;              // positions 0 .. before - 1 have left the window
  return a.pool > 0 ? before / a.pool : min(a.keep_first, before);
}
__device__ __forceinline__ int window_lo(const AttnBiasArgs& a, int i) {
  const int lo = a.chunk > 0 ? (i / a.chunk) * a.chunk : 0;
  return a.window > 0 ? max(lo, i - a.window + 1) : lo;
}
// the cache row of prefix key u of a request (pooled caches when pool > 0)
__device__ __forceinline__ int64_t prefix_row(const AttnBiasArgs& a, const int32_t* bt, int g, int u) {
  if (a.pool > 0) return ((int64_t)bt[u / a.pool_slots] * a.G + g) * a.pool_slots + u % a.pool_slots;
  return ((int64_t)bt[u / a.block_size] * a.G + g) * a.block_size + u % a.block_size;
}

// MAXV: value columns per lane
template <typename E, int MAXV>
__global__ void __launch_bounds__(ATT_WARPS * 32) attn_bias_chunk_kernel(AttnBiasArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float qs_all[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * ATT_WARPS + warp;
  if (item >= (int64_t)a.T * a.H) return;
  const int t = (int)(item / a.H), h = (int)(item % a.H);
  float* qs = qs_all + warp * a.dim;
  const E* q = (const E*)a.q + (int64_t)t * a.ldq + h * a.dim;
  for (int d = lane; d < a.dim; d += 32) qs[d] = ldf(q + d);
  __syncwarp();
  const int b = a.token_req[t], i = a.positions[t];
  const int lo = window_lo(a, i), npre = prefix_keys(a, i);
  const int g = h / (a.H / a.G);
  const float slope = a.bias_span > 0.f ? exp2f(-a.bias_span * (float)(h + 1) / (float)a.H) : 0.f;
  const int32_t* bt = a.block_table + (int64_t)b * a.max_blocks;
  const E* kc = (const E*)a.k_cache;
  const E* vc = (const E*)a.v_cache;
  const int64_t vld = a.v_ld > 0 ? a.v_ld : a.vdim;
  const bool pooled = a.pool > 0;
  const E* pkc = pooled ? (const E*)a.pk_cache : kc;
  const E* pvc = pooled ? (const E*)a.pv_cache : vc;
  float m = -INFINITY, l = 0.f, o[MAXV];
#pragma unroll
  for (int c = 0; c < MAXV; ++c) o[c] = 0.f;
  // the row's keys in one list: npre prefix keys, then positions lo .. i
  const int nkeys = npre + (i - lo + 1);
  for (int u0 = 0; u0 < nkeys; u0 += 32) {
    const int u = u0 + lane;
    const bool valid = u < nkeys, pre = u < npre;
    const int j = lo + (u - npre);
    int64_t row = 0;
    float s = -INFINITY;
    if (valid) {
      row = pre ? prefix_row(a, bt, g, u) : ((int64_t)bt[j / a.block_size] * a.G + g) * a.block_size + j % a.block_size;
      const E* kr = (pre ? pkc : kc) + row * a.dim;
      float acc = 0.f;
      for (int d = 0; d < a.dim; ++d) acc = fmaf(qs[d], ldf(kr + d), acc);
      acc *= a.scale;
      if (a.softcap > 0.f) acc = a.softcap * tanhf(acc / a.softcap);
      s = pre ? acc : acc - slope * (float)(i - j);
    }
    const float mn = fmaxf(m, warp_max(s));
    const float p = valid ? expf(s - mn) : 0.f;
    const float corr = expf(m - mn);            // m = -inf on the first tile: exp(-inf) = 0
    l = l * corr + warp_sum(p);
    m = mn;
#pragma unroll
    for (int c = 0; c < MAXV; ++c) o[c] *= corr;
    const int cnt = min(32, nkeys - u0);
    for (int jj = 0; jj < cnt; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const int64_t rj = __shfl_sync(0xffffffffu, row, jj);
      const E* vr = (u0 + jj < npre ? pvc : vc) + rj * vld;
#pragma unroll
      for (int c = 0; c < MAXV; ++c) {
        const int col = c * 32 + lane;
        if (col < a.vdim) o[c] = fmaf(pj, ldf(vr + col), o[c]);
      }
    }
  }
  if (a.sinks) {                                // the sink logit joins the denominator: no key, no value
    const float sk = a.sinks[h], mn = fmaxf(m, sk), corr = expf(m - mn);
    l = l * corr + expf(sk - mn);
#pragma unroll
    for (int c = 0; c < MAXV; ++c) o[c] *= corr;
  }
  const float inv = a.out_scale / l;
  E* out = (E*)a.out + (int64_t)t * a.ldo + h * a.vdim;
#pragma unroll
  for (int c = 0; c < MAXV; ++c) {
    const int col = c * 32 + lane;
    if (col < a.vdim) stf(out + col, o[c] * inv);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// bfloat16, head sizes that are multiples of 16 (keys) / 8 (values) up to 128: the same attention on the tensor cores
// (mma.sync m16n8k16).  A CTA owns 16 rows - consecutive (token, query head of one key/value head) pairs of one
// request, so neighbouring tokens and the heads of a group share every key tile - and its four warps take the 32-key
// tiles of the rows' chunk in turn: K and V of a tile are staged in the warp's own shared memory with 16-byte loads,
// S = Q K^T and O += P V are mma instructions with fp32 accumulators, bias, mask and softmax statistics stay in fp32,
// and the four partial results (m, l, O) are merged through shared memory at the end.  Decoding a single token is the
// same kernel with hpg rows in use: its four warps split the chunk's keys.
constexpr int AM_WARPS = 4, AM_KT = 32, AM_MAXD = 128, AM_PAD = 8;

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// tanh(x) = 1 - 2 / (e^(2x) + 1): absolute error of a few 1e-7 over the whole range (saturates cleanly at +-1)
__device__ __forceinline__ float tanh_fast(float x) {
  return 1.f - __fdividef(2.f, exp2f(fminf(x * 2.8853900817779268f, 100.f)) + 1.f);
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&p);
}

__device__ __forceinline__ void ab_ldsm(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ab_ldsm_t(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}

// ROWS = false: a CTA owns 16 rows and its warps split the key tiles (decoding, short pieces); where that leaves most of the chip idle,
// the warps of a cluster do, and its CTAs' sums meet over distributed shared memory.  A tile's keys and values are asked for at once
// (cp.async): with a round trip per eight pieces and one CTA per (request, group) two requests of 1160 keys in chunks of 1024 took 27 us
// (cold caches), 14.5 with clusters of eight.  ROWS = true: a CTA owns 64 rows, 16 per warp, and every key tile is staged once for all four warps (prompts).
// AHEAD (one row a request): what is there before the step - positions, block ids and a warp's first tile, all keys but the last - is
// fetched while the kernels before still run; only q and the last key wait for them.  With the states of the recurrences likewise, a
// decode step of a 2048-wide design (four layers, two of each mixer, two requests of 1160 keys) 311 us before and 297 so.
template <bool ROWS, bool AHEAD = false>
__global__ void __launch_bounds__(AM_WARPS * 32) attn_bias_mma_kernel(AttnBiasArgs a, int req0) {
  pdl_launch_dependents();
  if (!AHEAD) pdl_wait();
  typedef __nv_bfloat16 E;
  extern __shared__ __align__(16) unsigned char am_smem[];
  // CTAs of a cluster (1 or more; ROWS: 1) share the rows
  const int S = ROWS ? 1 : (int)cluster_nctarank(), crank = ROWS ? 0 : (int)cluster_ctarank();
  const int b = req0 + blockIdx.z, g = blockIdx.y, hpg = a.H / a.G;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qr = lane >> 2, qc = (lane & 3) * 2;
  const int rs = a.qsl[b], nrows = (a.qsl[b + 1] - rs) * hpg, Rc = (int)(blockIdx.x / S) * (ROWS ? 16 * AM_WARPS : 16);
  if (Rc >= nrows) return;
  const int R0 = ROWS ? Rc + warp * 16 : Rc;               // may lie beyond the request's rows: such a warp only helps staging
  const int dim = a.dim, vdim = a.vdim, ksteps = dim >> 4, vtiles = vdim >> 3;
  const int kst = dim + AM_PAD, vst = vdim + AM_PAD;                 // shared row strides (elements)
  const size_t region = (size_t)AM_KT * (kst + vst) * sizeof(E);
  E* Ks = reinterpret_cast<E*>(am_smem + (ROWS ? 0 : warp) * region);
  E* Vs = Ks + AM_KT * kst;
  // this thread's two rows: qr and qr + 8 of the tile
  int pos[2], lo[2], tok[2], head[2], npre[2];
  float slope2[2];
  const float log2e = 1.4426950408889634f;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = R0 + qr + 8 * h;
    const bool valid = r < nrows;
    tok[h] = rs + (valid ? r : nrows - 1) / hpg;
    head[h] = g * hpg + (valid ? r : nrows - 1) % hpg;
    pos[h] = valid ? a.positions[tok[h]] : -1;                       // -1: no key is visible, the row is never written
    lo[h] = pos[h] >= 0 ? window_lo(a, pos[h]) : 0;
    npre[h] = pos[h] >= 0 ? prefix_keys(a, pos[h]) : 0;
    slope2[h] = a.bias_span > 0.f ? exp2f(-a.bias_span * (float)(head[h] + 1) / (float)a.H) * log2e : 0.f;
  }
  const int pos_first = a.positions[rs + Rc / hpg], pos_last = a.positions[rs + min(Rc + (ROWS ? 16 * AM_WARPS : 16) - 1, nrows - 1) / hpg];
  const int lo_min = window_lo(a, pos_first);
  // prefix keys (kept first tokens or pooled blocks) come first, in tiles of their own; the last row of the CTA sees the most
  const int pre_cta = prefix_keys(a, pos_last), ptiles = (pre_cta + AM_KT - 1) / AM_KT;
  const int ntiles = ptiles + (pos_last - lo_min + AM_KT) / AM_KT;
  // the keys this warp's own rows can see (ROWS: tiles outside are staged for the others but not computed here)
  // (the same for every lane of the warp: the mma instructions below need all 32 lanes on one path)
  const bool wany = R0 < nrows;
  const int own_hi = wany ? a.positions[rs + min(R0 + 15, nrows - 1) / hpg] : -1;
  const int own_first = wany ? a.positions[rs + R0 / hpg] : 0;
  const int own_lo = window_lo(a, own_first), own_pre = wany ? prefix_keys(a, own_hi) : 0;
  const float scale2 = a.scale * log2e;
  const float cap2 = a.softcap * log2e, cap_in = a.softcap > 0.f ? a.scale / a.softcap : 0.f;   // capped scores, in units of log 2
  uint32_t qf[AM_MAXD / 16][4];
  auto load_q = [&]() {
#pragma unroll
    for (int ks = 0; ks < AM_MAXD / 16; ++ks) {
      if (ks < ksteps) {
        const E* q0 = (const E*)a.q + (int64_t)tok[0] * a.ldq + head[0] * dim + ks * 16 + qc;
        const E* q1 = (const E*)a.q + (int64_t)tok[1] * a.ldq + head[1] * dim + ks * 16 + qc;
        qf[ks][0] = pos[0] >= 0 ? *reinterpret_cast<const uint32_t*>(q0) : 0u;
        qf[ks][1] = pos[1] >= 0 ? *reinterpret_cast<const uint32_t*>(q1) : 0u;
        qf[ks][2] = pos[0] >= 0 ? *reinterpret_cast<const uint32_t*>(q0 + 8) : 0u;
        qf[ks][3] = pos[1] >= 0 ? *reinterpret_cast<const uint32_t*>(q1 + 8) : 0u;
      } else {
        qf[ks][0] = qf[ks][1] = qf[ks][2] = qf[ks][3] = 0u;
      }
    }
  };
  if (!AHEAD) load_q();
  float o[AM_MAXD / 8][4];
#pragma unroll
  for (int v = 0; v < AM_MAXD / 8; ++v) o[v][0] = o[v][1] = o[v][2] = o[v][3] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  const int32_t* bt = a.block_table + (int64_t)b * a.max_blocks;
  const int kseg = dim >> 3, vseg = vdim >> 3, vld = a.v_ld > 0 ? a.v_ld : vdim;
  const int kt_first = ROWS ? 0 : crank * AM_WARPS + warp;
  // where key j0 + lane of a tile lives (-1: nowhere)
  auto row_at = [&](bool ptile, int j0) -> int64_t {
    const int jl = j0 + lane;
    if (ptile) return jl < pre_cta ? prefix_row(a, bt, g, jl) : -1;
    return jl <= pos_last ? ((int64_t)bt[jl / a.block_size] * a.G + g) * a.block_size + jl % a.block_size : -1;
  };
  // a tile's keys and values for one warp: the 16-byte pieces of a row are fetched by consecutive lanes (whole warps run the loops: the
  // shuffle needs every lane); key `skip` is left out
  auto stage = [&](E* dst, const E* src, int segs, int st, int64_t ld, int64_t myrow, int skip) {
    for (int idx = lane; idx < AM_KT * segs; idx += 32) {
      const int key = idx / segs, seg = idx % segs;
      const int64_t row = __shfl_sync(0xffffffffu, myrow, key);
      asm volatile("{\n.reg .pred p;\nsetp.eq.u32 p, %3, 0;\n@p cp.async.cg.shared.global [%0], [%1], 16, %2;\n}" ::"r"((uint32_t)__cvta_generic_to_shared(dst + key * st + seg * 8)),
                   "l"(src + (row >= 0 ? row * ld + seg * 8 : 0)), "r"(row >= 0 ? 16 : 0), "r"((uint32_t)(AHEAD && key == skip)) : "memory");
    }
  };
  if constexpr (AHEAD) {
    const int j0 = lo_min + kt_first * AM_KT, own = pos_last - j0;      // (no prefix keys here)
    const E* kc = (const E*)a.k_cache;
    const E* vc = (const E*)a.v_cache;
    int64_t myrow = -1;
    if (kt_first < ntiles) {
      myrow = row_at(false, j0);
      stage(Ks, kc, kseg, kst, dim, myrow, own);
      stage(Vs, vc, vseg, vst, vld, myrow, own);
    }
    pdl_wait();
    load_q();
    if (kt_first < ntiles && own < AM_KT) {
      const int64_t row = __shfl_sync(0xffffffffu, myrow, own);
      for (int i = lane; i < kseg + vseg; i += 32) {
        const bool key = i < kseg;
        const int seg = key ? i : i - kseg;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared((key ? Ks + own * kst : Vs + own * vst) + seg * 8)),
                     "l"((key ? kc + row * dim : vc + row * vld) + seg * 8) : "memory");
      }
    }
  }
  for (int kt = kt_first; kt < ntiles; kt += ROWS ? 1 : AM_WARPS * S) {
    const bool ptile = kt < ptiles;                         // a tile of prefix keys: j0 counts them from 0
    const int j0 = ptile ? kt * AM_KT : lo_min + (kt - ptiles) * AM_KT;
    const E* kc = (const E*)(ptile && a.pool > 0 ? a.pk_cache : a.k_cache);
    const E* vc = (const E*)(ptile && a.pool > 0 ? a.pv_cache : a.v_cache);
    if (ROWS) __syncthreads();                              // the previous tile has been read by every warp
    int64_t myrow = -1;
    if (!AHEAD || kt != kt_first) myrow = row_at(ptile, j0);
    if constexpr (!ROWS) {
      if (!AHEAD || kt != kt_first) {
        stage(Ks, kc, kseg, kst, dim, myrow, -1);
        stage(Vs, vc, vseg, vst, vld, myrow, -1);
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    } else {
      // four 16-byte pieces are requested before the first is stored, so a tile costs a few memory round trips, not one per piece
      constexpr int SU = 4, sstep = AM_WARPS * 32;
      for (int idx0 = 0; idx0 < AM_KT * kseg; idx0 += SU * sstep) {
        uint4 v[SU]; int dst[SU];
#pragma unroll
        for (int u = 0; u < SU; ++u) {
          const int idx = min(idx0 + u * sstep + (int)threadIdx.x, AM_KT * kseg - 1);
          const int key = idx / kseg, seg = idx % kseg;
          const int64_t row = __shfl_sync(0xffffffffu, myrow, key);
          v[u] = make_uint4(0u, 0u, 0u, 0u);
          if (row >= 0) v[u] = *reinterpret_cast<const uint4*>(kc + row * dim + seg * 8);
          dst[u] = key * kst + seg * 8;
        }
#pragma unroll
        for (int u = 0; u < SU; ++u) *reinterpret_cast<uint4*>(Ks + dst[u]) = v[u];
      }
      for (int idx0 = 0; idx0 < AM_KT * vseg; idx0 += SU * sstep) {
        uint4 v[SU]; int dst[SU];
#pragma unroll
        for (int u = 0; u < SU; ++u) {
          const int idx = min(idx0 + u * sstep + (int)threadIdx.x, AM_KT * vseg - 1);
          const int key = idx / vseg, seg = idx % vseg;
          const int64_t row = __shfl_sync(0xffffffffu, myrow, key);
          v[u] = make_uint4(0u, 0u, 0u, 0u);
          if (row >= 0) v[u] = *reinterpret_cast<const uint4*>(vc + row * vld + seg * 8);
          dst[u] = key * vst + seg * 8;
        }
#pragma unroll
        for (int u = 0; u < SU; ++u) *reinterpret_cast<uint4*>(Vs + dst[u]) = v[u];
      }
    }
    if (ROWS) __syncthreads(); else __syncwarp();
    if (ROWS && (ptile ? j0 >= own_pre : (j0 > own_hi || j0 + AM_KT <= own_lo))) continue;
    float sacc[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) sacc[nt][0] = sacc[nt][1] = sacc[nt][2] = sacc[nt][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < AM_MAXD / 16; ++ks) {
      if (ks < ksteps) {
#pragma unroll
        for (int nt = 0; nt < 4; nt += 2) {
          uint32_t kf[4];                                    // keys nt * 8 .. + 15, both halves of the 16 dimensions
          ab_ldsm(kf, Ks + (nt * 8 + (lane & 7) + ((lane >> 4) & 1) * 8) * kst + ks * 16 + ((lane >> 3) & 1) * 8);
          mma_16816(sacc[nt], qf[ks], kf[0], kf[1]);
          mma_16816(sacc[nt + 1], qf[ks], kf[2], kf[3]);
        }
      }
    }
    // bias, mask, running maximum (exponent base 2)
    float tmax[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int h = c >> 1, j = j0 + nt * 8 + qc + (c & 1);
        const bool vis = ptile ? j < npre[h] : (j <= pos[h] && j >= lo[h]);
        float sc = sacc[nt][c] * scale2;
        if (cap2 > 0.f) sc = cap2 * tanh_fast(sacc[nt][c] * cap_in);
        const float sv = vis ? (ptile ? sc : sc - slope2[h] * (float)(pos[h] - j)) : -INFINITY;
        sacc[nt][c] = sv;
        tmax[h] = fmaxf(tmax[h], sv);
      }
    float corr[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      tmax[h] = fmaxf(tmax[h], __shfl_xor_sync(0xffffffffu, tmax[h], 1));
      tmax[h] = fmaxf(tmax[h], __shfl_xor_sync(0xffffffffu, tmax[h], 2));
      const float mn = fmaxf(m[h], tmax[h]);
      corr[h] = mn == -INFINITY ? 1.f : exp2f(m[h] - mn);
      m[h] = mn;
      l[h] *= corr[h];
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int h = c >> 1;
        const float p = sacc[nt][c] == -INFINITY ? 0.f : exp2f(sacc[nt][c] - m[h]);
        sacc[nt][c] = p;
        l[h] += p;
      }
#pragma unroll
    for (int v = 0; v < AM_MAXD / 8; ++v) { o[v][0] *= corr[0]; o[v][1] *= corr[0]; o[v][2] *= corr[1]; o[v][3] *= corr[1]; }
    uint32_t pf[2][4];
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      pf[kk][0] = pack2(sacc[2 * kk][0], sacc[2 * kk][1]);
      pf[kk][1] = pack2(sacc[2 * kk][2], sacc[2 * kk][3]);
      pf[kk][2] = pack2(sacc[2 * kk + 1][0], sacc[2 * kk + 1][1]);
      pf[kk][3] = pack2(sacc[2 * kk + 1][2], sacc[2 * kk + 1][3]);
    }
#pragma unroll
    for (int v = 0; v < AM_MAXD / 8; v += 2) {
      if (v < vtiles) {
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          uint32_t vf[4];                                    // 16 keys x 16 columns (an odd last tile reads the row's padding)
          ab_ldsm_t(vf, Vs + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * vst + v * 8 + (lane >> 4) * 8);
          mma_16816(o[v], pf[kk], vf[0], vf[1]);
          if (v + 1 < vtiles) mma_16816(o[v + 1], pf[kk], vf[2], vf[3]);
        }
      }
    }
    if (!ROWS) __syncwarp();
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
  }
  if (ROWS) {
    // each warp finished its own rows: normalise and store from the registers
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (pos[h] < 0) continue;
      float oc = 1.f;
      if (a.sinks) {
        const float sk = a.sinks[head[h]] * log2e, mn = fmaxf(m[h], sk);
        oc = exp2f(m[h] - mn);
        l[h] = l[h] * oc + exp2f(sk - mn);
      }
      const float inv = a.out_scale * oc / l[h];
      E* out = (E*)a.out + (int64_t)tok[h] * a.ldo + head[h] * vdim + qc;
#pragma unroll
      for (int v = 0; v < AM_MAXD / 8; ++v)
        if (v < vtiles) *reinterpret_cast<uint32_t*>(out + v * 8) = pack2(o[v][2 * h] * inv, o[v][2 * h + 1] * inv);
    }
    return;
  }
  // merge the four warps' partial results
  __syncthreads();                                          // every warp is done with its tiles: the regions are free
  float* Os = reinterpret_cast<float*>(am_smem + warp * region);      // [16][vdim]
  float* ML = reinterpret_cast<float*>(am_smem + AM_WARPS * region);  // [warps][2][16]
#pragma unroll
  for (int v = 0; v < AM_MAXD / 8; ++v) {
    if (v < vtiles) {
      Os[qr * vdim + v * 8 + qc] = o[v][0]; Os[qr * vdim + v * 8 + qc + 1] = o[v][1];
      Os[(qr + 8) * vdim + v * 8 + qc] = o[v][2]; Os[(qr + 8) * vdim + v * 8 + qc + 1] = o[v][3];
    }
  }
  if ((lane & 3) == 0) {
    ML[(warp * 2 + 0) * 16 + qr] = m[0]; ML[(warp * 2 + 0) * 16 + qr + 8] = m[1];
    ML[(warp * 2 + 1) * 16 + qr] = l[0]; ML[(warp * 2 + 1) * 16 + qr + 8] = l[1];
  }
  __syncthreads();
  // a row's largest score and, relative to it, its sums: over this CTA's warps, then over the cluster's CTAs in rank order
  auto finish = [&](int r, int c, float M, auto&& sums) {
    const int row = R0 + r;
    float num = 0.f, den = 0.f;
    if (a.sinks) {
      const float sk = a.sinks[g * hpg + row % hpg] * log2e;
      M = fmaxf(M, sk);
      den = exp2f(sk - M);
    }
    sums(M, num, den);
    E* out = (E*)a.out + (int64_t)(rs + row / hpg) * a.ldo + (g * hpg + row % hpg) * vdim + c;
    *out = __float2bfloat16_rn(num / den * a.out_scale);
  };
  auto warps_max = [&](int r) {
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < AM_WARPS; ++w) M = fmaxf(M, ML[(w * 2) * 16 + r]);
    return M;
  };
  auto warps_sum = [&](int r, int c, float M, float& num, float& den) {
#pragma unroll
    for (int w = 0; w < AM_WARPS; ++w) {
      const float mw = ML[(w * 2) * 16 + r];
      const float f = mw == -INFINITY ? 0.f : exp2f(mw - M);
      num = fmaf(f, reinterpret_cast<const float*>(am_smem + w * region)[r * vdim + c], num);
      den = fmaf(f, ML[(w * 2 + 1) * 16 + r], den);
    }
  };
  if (S == 1) {
    for (int idx = threadIdx.x; idx < 16 * vdim; idx += AM_WARPS * 32) {
      const int r = idx / vdim, c = idx % vdim;
      if (R0 + r >= nrows) continue;
      finish(r, c, warps_max(r), [&](float M, float& num, float& den) { warps_sum(r, c, M, num, den); });
    }
    return;
  }
  float* part = ML + AM_WARPS * 2 * 16;                     // this CTA's sums: [16][vdim], then [2][16]: largest scores, weights
  for (int idx = threadIdx.x; idx < 16 * vdim; idx += AM_WARPS * 32) {
    const int r = idx / vdim, c = idx % vdim;
    const float M = warps_max(r);
    float num = 0.f, den = 0.f;
    if (M != -INFINITY) warps_sum(r, c, M, num, den);
    part[idx] = num;
    if (c == 0) { part[16 * vdim + r] = M; part[16 * vdim + 16 + r] = den; }
  }
  cluster_arrive();                                         // every CTA's sums are in its shared memory
  cluster_wait();
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(part);
  auto remote = [&](int rank, int i) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(mapa_u32(mine + i * 4, (uint32_t)rank)) : "memory");
    return v;
  };
  for (int idx = crank * AM_WARPS * 32 + threadIdx.x; idx < 16 * vdim; idx += S * AM_WARPS * 32) {
    const int r = idx / vdim, c = idx % vdim;
    if (R0 + r >= nrows) continue;
    float mr[8], M = -INFINITY;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      mr[k] = k < S ? remote(k, 16 * vdim + r) : -INFINITY;
      M = fmaxf(M, mr[k]);
    }
    finish(r, c, M, [&](float Mall, float& num, float& den) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < S) {
          const float f = mr[k] == -INFINITY ? 0.f : exp2f(mr[k] - Mall);
          num = fmaf(f, remote(k, idx), num);
          den = fmaf(f, remote(k, 16 * vdim + 16 + r), den);
        }
    });
  }
  cluster_arrive();                                         // nobody leaves while a peer reads its sums
  cluster_wait();
}

// CTAs per cluster for `ctas` CTAs whose rows see up to `tiles` key tiles: as many as a round of one CTA per SM has room for, while each
// warp keeps a tile
static int bias_cluster(int64_t ctas, int tiles) {
  int S = 8;
  while (S > 1 && (ctas * S > 148 || tiles < AM_WARPS * S)) S /= 2;
  return S;
}
static cudaError_t launch_bias_split(dim3 grid, int S, size_t smem, cudaStream_t st, const AttnBiasArgs& a, int req0) {
  grid.x *= S;
  // pooled blocks may be written in the step, and the first tokens of a window are tiles of their own
  auto kern = req0 == 0 && a.max_q == 1 && a.keys_before && a.pool == 0 && a.keep_first == 0 ? attn_bias_mma_kernel<false, true> : attn_bias_mma_kernel<false>;
  if (S == 1) return launch_pdl(kern, grid, dim3(AM_WARPS * 32), smem, st, a, req0);
  prefer_max_shared(kern);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(AM_WARPS * 32); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl_for_this_launch() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, a, req0);
}

inline namespace KGE_ELT_NS {
int paged_attn_bias_pair(void* out, int ldo, const void* q, int ldq, const void* kc, const void* vc, const int32_t* bt, int max_blocks, const int32_t* sl,
                         const int32_t* qsl, int B, int T, int max_q_len, int max_seq_len, int H, int KV, int hd, int bs, float scale, int chunk, float span, float out_scale, cudaStream_t st);      // attn_tc.cu
}
// What the tcgen05 kernel of attn_pair.cuh takes: plain chunked attention with distance biases, keys and values of 64 or 128, pages of a
// power of two of at least 8 tokens, aligned rows.  Two prompts of 1150 tokens, 16 / 4 heads of 128 in chunks of 1024: 162 us in the
// kernel above, 34 there.
static bool bias_pair_ok(const AttnBiasArgs& a) {
  return a.elt == KGE_ELT_BF16 && (a.dim == 64 || a.dim == 128) && a.vdim == a.dim && (a.v_ld == 0 || a.v_ld == a.vdim) && a.softcap == 0.f && !a.sinks && a.window == 0 &&
         a.seq_lens && a.H % a.G == 0 && a.H / a.G <= 128 && a.block_size >= 8 && (a.block_size & (a.block_size - 1)) == 0 && a.ldq % 8 == 0 && a.ldo % 8 == 0 && a.scale > 0.f &&
         ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.k_cache) | reinterpret_cast<uintptr_t>(a.v_cache)) & 15) == 0;
}

int attn_bias_chunk(const AttnBiasArgs& a, cudaStream_t st) {
  if (a.T <= 0) return 0;
  KGE_REQUIRE(a.window >= 0 && (a.window > 0 || (a.keep_first == 0 && a.pool == 0)) && !(a.keep_first > 0 && a.pool > 0) && (a.window == 0 || a.bias_span == 0.f) &&
              (a.pool == 0 || (a.pk_cache && a.pv_cache && a.pool_slots > 0)),
              "attn_bias_chunk: window %d with %d kept tokens / pooled blocks of %d", a.window, a.keep_first, a.pool);
  if (a.elt == KGE_ELT_BF16 && a.max_q > 0 && a.dim % 16 == 0 && a.dim <= AM_MAXD && a.vdim % 8 == 0 && a.vdim <= AM_MAXD && a.ldq % 2 == 0 &&
      a.H % a.G == 0 && a.v_ld % 8 == 0 && (reinterpret_cast<uintptr_t>(a.q) & 3) == 0 && a.B <= 65535 && a.G <= 65535) {
    const int hpg = a.H / a.G;
    // a tile for all warps (ROWS), or one each, their statistics and, in a cluster, the CTA's sums
    auto tile_of = [](int dim, int vdim) { return (size_t)AM_KT * (dim + vdim + 2 * AM_PAD) * 2; };
    auto split_of = [&](int dim, int vdim) { return AM_WARPS * tile_of(dim, vdim) + (size_t)AM_WARPS * 2 * 16 * 4; };
    auto sums_of = [](int vdim) { return (size_t)16 * (vdim + 2) * 4; };
    const size_t tile = tile_of(a.dim, a.vdim), split = split_of(a.dim, a.vdim), sums = sums_of(a.vdim);
    // the function's limit on this device, for every size
    if (split + sums > 48 * 1024)
      for (auto kern : {attn_bias_mma_kernel<false>, attn_bias_mma_kernel<false, true>})
        KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(split_of(AM_MAXD, AM_MAXD) + sums_of(AM_MAXD))));
    // the leading one-token requests, then the rest; 64-row CTAs where a request has that many rows and its output
    // pairs can be stored as 32-bit words
    const int D = std::min(std::max(a.num_decode, 0), a.B);
    // the keys of a row that the launch can know of: its chunk, its window, or the block table's reach
    const int reach = std::min(a.max_blocks * a.block_size, a.window > 0 ? a.window + a.keep_first : a.chunk > 0 ? a.chunk : 1 << 30);
    if (D > 0) {
      const int S = bias_cluster((int64_t)((hpg + 15) / 16) * a.G * D, reach / AM_KT);
      KGE_CUDA_OK(launch_bias_split(dim3((hpg + 15) / 16, a.G, D), S, S > 1 ? split + sums : split, st, a, 0));
    }
    // the tcgen05 kernel's start shows where all keys are one tile of this kernel: 32 / 8 heads of 128, one piece of 9 tokens 6.25 us here and 7.2
    // there, of 32 7.1 and 7.4, eight of 17 7.1 and 7.4 (eight of 20 behind 8 keys 8.9 and 7.6, heads of 64 level)
    const int max_seq = a.max_seq > 0 ? a.max_seq : (int)std::min<int64_t>((int64_t)a.max_blocks * a.block_size, INT32_MAX);
    if (D < a.B && a.max_q * hpg > 32 && max_seq > AM_KT && bias_pair_ok(a))
      return paged_attn_bias_pair(a.out, a.ldo, a.q, a.ldq, a.k_cache, a.v_cache, a.block_table + (int64_t)D * a.max_blocks, a.max_blocks, a.seq_lens + D, a.qsl + D, a.B - D, a.T - D,
                                  a.max_q, max_seq, a.H, a.G, a.dim, a.block_size, a.scale, a.chunk, a.bias_span, a.out_scale, st);
    if (D < a.B) {
      const int rows = a.max_q * hpg;
      const bool wide = rows > 32 && a.ldo % 2 == 0 && a.vdim % 2 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 3) == 0;
      if (wide) KGE_CUDA_OK(launch_pdl(attn_bias_mma_kernel<true>, dim3((rows + 16 * AM_WARPS - 1) / (16 * AM_WARPS), a.G, a.B - D), dim3(AM_WARPS * 32), tile, st, a, D));
      else KGE_CUDA_OK(launch_bias_split(dim3((rows + 15) / 16, a.G, a.B - D), 1, split, st, a, D));
    }
    return 0;
  }
  KGE_REQUIRE(a.vdim <= 32 * ATT_MAXV, "attn_bias_chunk: value head size %d > %d", a.vdim, 32 * ATT_MAXV);
  KGE_REQUIRE(a.dim <= 2048 && a.H % a.G == 0, "attn_bias_chunk: bad head sizes");
  const int64_t items = (int64_t)a.T * a.H;
  const dim3 grid((unsigned)((items + ATT_WARPS - 1) / ATT_WARPS)), block(ATT_WARPS * 32);
  const size_t smem = (size_t)ATT_WARPS * a.dim * 4;
  cudaError_t ce;
  const bool f32 = a.elt == KGE_ELT_F32;
  if (a.vdim <= 256) ce = f32 ? launch_pdl(attn_bias_chunk_kernel<float, 8>, grid, block, smem, st, a) : launch_pdl(attn_bias_chunk_kernel<__nv_bfloat16, 8>, grid, block, smem, st, a);
  else ce = f32 ? launch_pdl(attn_bias_chunk_kernel<float, ATT_MAXV>, grid, block, smem, st, a) : launch_pdl(attn_bias_chunk_kernel<__nv_bfloat16, ATT_MAXV>, grid, block, smem, st, a);
  KGE_CUDA_OK(ce);
  return 0;
}

// W: numbers per thread and pass, 16 bytes of them where rows, heads and caches allow
template <typename E, int W>
__global__ void kv_write_any_kernel(const E* k, int ldk, const E* v, int ldv, const int64_t* slots, E* kc, E* vc, int G, int dim, int vdim, int bs) {
  struct __align__(W * sizeof(E)) Piece { E e[W]; };
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const int64_t slot = slots[t];
  if (slot < 0) return;
  const int64_t blk = slot / bs, off = slot % bs;
  const int nk = G * dim / W, n = nk + G * vdim / W;          // keys, then values
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const bool key = i < nk;
    const int c = (key ? i : i - nk) * W, hd = key ? dim : vdim, g = c / hd, d = c % hd;
    const E* src = (key ? k + (int64_t)t * ldk : v + (int64_t)t * ldv) + c;
    E* dst = (key ? kc : vc) + ((blk * G + g) * bs + off) * hd + d;
    *reinterpret_cast<Piece*>(dst) = *reinterpret_cast<const Piece*>(src);
  }
}

template <typename E, int W>
static cudaError_t launch_kv_write(const void* k, int ldk, const void* v, int ldv, const int64_t* slots, void* kc, void* vc, int T, int G, int dim, int vdim, int bs, cudaStream_t st) {
  const int n = (G * dim + G * vdim) / W, th = std::max(32, std::min(256, (n + 31) / 32 * 32));
  return launch_pdl(kv_write_any_kernel<E, W>, dim3(T), dim3(th), 0, st, (const E*)k, ldk, (const E*)v, ldv, slots, (E*)kc, (E*)vc, G, dim, vdim, bs);
}
int kv_write_any(const void* k, int ldk, const void* v, int ldv, const int64_t* slots, void* k_cache, void* v_cache, int T, int G,
                 int dim, int vdim, int block_size, int elt, cudaStream_t st) {
  if (T <= 0) return 0;
  const int per = elt == KGE_ELT_F32 ? 4 : 8;
  const bool wide = dim % per == 0 && vdim % per == 0 && ldk % per == 0 && ldv % per == 0 &&
                    ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) == 0;
  auto run = elt == KGE_ELT_F32 ? (wide ? launch_kv_write<float, 4> : launch_kv_write<float, 1>)
                                : (wide ? launch_kv_write<__nv_bfloat16, 8> : launch_kv_write<__nv_bfloat16, 1>);
  KGE_CUDA_OK(run(k, ldk, v, ldv, slots, k_cache, v_cache, T, G, dim, vdim, block_size, st));
  return 0;
}

// One block per (token, key/value head); only a token that ends a block of `pool` positions has work: the block's keys
// and values are read back from the caches (so what is averaged is what the attention reads), sixteen rows requested at a
// time, summed in fp32 in ascending position and divided by the count.  One column per thread and pass.
template <typename E>
__global__ void __launch_bounds__(256) pool_kv_write_kernel(PoolKvArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, g = blockIdx.y, pos = a.positions[t];
  if ((pos + 1) % a.pool != 0) return;
  const int pb = pos / a.pool, p0 = pb * a.pool;
  const int32_t* bt = a.block_table + (int64_t)a.token_req[t] * a.max_blocks;
  const int64_t drow = ((int64_t)bt[pb / a.pool_slots] * a.G + g) * a.pool_slots + pb % a.pool_slots;
  for (int c = threadIdx.x; c < a.dim + a.vdim; c += blockDim.x) {
    const bool isk = c < a.dim;
    const int w = isk ? a.dim : a.vdim, dd = isk ? c : c - a.dim;
    const E* src = (const E*)(isk ? a.k_cache : a.v_cache);
    float acc = 0.f;
    for (int j0 = p0; j0 <= pos; j0 += 16) {
      float v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int j = j0 + u;
        v[u] = j <= pos ? ldf(src + (((int64_t)bt[j / a.block_size] * a.G + g) * a.block_size + j % a.block_size) * w + dd) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) acc += v[u];
    }
    E* dst = (E*)(isk ? a.pk_cache : a.pv_cache);
    stf(dst + drow * w + dd, acc / (float)a.pool);
  }
}

int pool_kv_write(const PoolKvArgs& a, cudaStream_t st) {
  if (a.T <= 0) return 0;
  KGE_REQUIRE(a.pool >= 1 && a.pool_slots >= 1 && a.pool_slots * a.pool >= a.block_size && a.G <= 65535, "pool_kv_write: blocks of %d positions, %d entries per page of %d", a.pool, a.pool_slots, a.block_size);
  cudaError_t ce = a.elt == KGE_ELT_F32 ? launch_pdl(pool_kv_write_kernel<float>, dim3(a.T, a.G), dim3(256), 0, st, a)
                                        : launch_pdl(pool_kv_write_kernel<__nv_bfloat16>, dim3(a.T, a.G), dim3(256), 0, st, a);
  KGE_CUDA_OK(ce);
  return 0;
}

}  // namespace kge
