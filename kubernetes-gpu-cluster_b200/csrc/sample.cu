// Temperature / top-k / top-p sampling, no sort.  A row belongs to a thread-block cluster; its CTAs hold the row's 16-bit
// logits in shared memory (as order-preserving integers) from one read of HBM / L2 on, and every search step is a pass over
// shared memory, a warp reduction and one exchange over distributed shared memory:
//   top-k   the k-th largest key by counts, an interval of keys cut in eight per step; first among the threads' largest keys,
//           which bounds it from below, so that the steps over all elements visit few of them;
//   top-p   the smallest key whose mass from below exceeds 1 - p, an interval cut in four per step, by softmax mass (fp32,
//           summed in a fixed order); a step visits the elements inside the interval only;
//   draw    the Gumbel-max form the reference uses, argmax(p_i / q_i) with q ~ Exp(1), over the kept set.
// What bounds it: instruction issue of the exponentials and of Philox (ten rounds per kept element), and the chain of 6 to 12
// cluster exchanges (1 to 2 us each); the one read of V * 2 bytes is about 2 us.  32 rows x 128256 on a B200, us:
// greedy 7, top-k 30, top-p 60, unfiltered 36, the four kinds in turn 51; one CTA per row with radix histograms in shared
// memory (counts and masses by atomics, four passes each over the row in L2 by 2-byte loads) took 1376 for those in turn.
#include <type_traits>

#include "common.cuh"
#include "kge.h"

namespace kge {
inline namespace KGE_ELT_NS {

constexpr int kSampleThreads = 512;

__device__ __forceinline__ uint32_t fkey(float f) {   // monotone: a < b  <=>  fkey(a) < fkey(b)
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Philox-4x32-10 -> one uniform in (0,1] per (seed, step, index)
__device__ __forceinline__ float philox_uniform(uint64_t seed, uint64_t step, uint32_t idx) {
  uint32_t c0 = idx, c1 = (uint32_t)step, c2 = (uint32_t)(step >> 32), c3 = 0x9E3779B9u;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0, n1 = (uint32_t)p1;
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1, n3 = (uint32_t)p0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
  return ((float)(c0 >> 8) + 1.0f) * (1.0f / 16777216.0f);
}

// The 16-bit logit as an integer key: a < b <=> key(a) < key(b); NaN sorts on top; 0 is no logit's key and marks "no element".
#ifdef KGE_HALF
constexpr uint32_t kNanBias = 0x03ff03ffu, kInfBits = 0x7c00u;
#else
constexpr uint32_t kNanBias = 0x007f007fu, kInfBits = 0x7f80u;
#endif
__device__ __forceinline__ uint32_t pack_keys(uint32_t u) {
  const uint32_t neg = (u >> 15) & 0x00010001u;
  uint32_t key = u ^ ((neg * 0xffffu) | 0x80008000u);
  if (((u & 0x7fff7fffu) + kNanBias) & 0x80008000u) {          // a NaN among the two
    if ((u & 0x7fffu) > kInfBits) key |= 0xffffu;
    if (((u >> 16) & 0x7fffu) > kInfBits) key |= 0xffff0000u;
  }
  return key;
}
__device__ __forceinline__ float key_value(uint32_t key) { return bf_lo((key & 0x8000u) ? key ^ 0x8000u : key ^ 0xffffu); }

__device__ __forceinline__ uint32_t value_key(float v) {      // the key of v rounded to the element type
  const bf16 h = f2bf(v);
  return pack_keys(*reinterpret_cast<const unsigned short*>(&h)) & 0xffffu;
}

__device__ __forceinline__ void st_cluster(const void* local, uint32_t rank, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(mapa_u32((uint32_t)__cvta_generic_to_shared(local), rank)), "r"(v) : "memory");
}

constexpr int kSampleWarps = kSampleThreads / 32;
constexpr int kMaxCluster = 8;

struct SampleShared {
  uint32_t warp[8][kSampleWarps];
  uint32_t all[2][kMaxCluster][8];       // what every CTA of the cluster contributed, two exchanges in flight
};

struct AddOp { template <typename T> __device__ __forceinline__ T operator()(T a, T b) const { return a + b; } };
struct MaxOp { template <typename T> __device__ __forceinline__ T operator()(T a, T b) const { return b > a ? b : a; } };

// Combine N <= 8 values over the cluster; every thread gets the results, combined in the same order everywhere.
template <int N, typename T, typename OP>
__device__ __forceinline__ void cluster_reduce(T (&v)[N], SampleShared& sh, int& phase, OP op) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t nc = cluster_nctarank();
#pragma unroll
  for (int k = 0; k < N; ++k) {
    if constexpr (std::is_same<T, int>::value && std::is_same<OP, AddOp>::value) {
      v[k] = __reduce_add_sync(0xffffffffu, v[k]);
    } else if constexpr (std::is_same<T, int>::value) {
      v[k] = __reduce_max_sync(0xffffffffu, v[k]);
    } else {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[k] = op(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    }
    if (lane == 0) sh.warp[k][wid] = *reinterpret_cast<uint32_t*>(&v[k]);
  }
  __syncthreads();
  if (wid < N) {
    uint32_t raw = sh.warp[wid][lane % kSampleWarps];
    T t = *reinterpret_cast<T*>(&raw);
#pragma unroll
    for (int o = kSampleWarps / 2; o > 0; o >>= 1) t = op(t, __shfl_xor_sync(0xffffffffu, t, o));
    if (lane < (int)nc) st_cluster(&sh.all[phase & 1][cluster_ctarank()][wid], lane, *reinterpret_cast<uint32_t*>(&t));
  }
  cluster_arrive(); cluster_wait();
  // lane (r, k) takes value k of ranks r and r + 4 (zero is neutral for the sums and for the maxima taken here)
  const int kk = lane & 7, r = lane >> 3;
  uint32_t raw = r < (int)nc && kk < N ? sh.all[phase & 1][r][kk] : 0u, raw4 = r + 4 < (int)nc && kk < N ? sh.all[phase & 1][r + 4][kk] : 0u;
  T t = op(*reinterpret_cast<T*>(&raw), *reinterpret_cast<T*>(&raw4));
  t = op(t, __shfl_xor_sync(0xffffffffu, t, 8));
  t = op(t, __shfl_xor_sync(0xffffffffu, t, 16));
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = __shfl_sync(0xffffffffu, t, k);
  ++phase;
}

// Eight consecutive logits as packed keys; elements beyond V are "no element".
__device__ __forceinline__ uint4 load_keys(const bf16* row, int v8, int V, bool aligned) {
  const int i = v8 * 8;
  if (aligned && i <= V - 8) {
    const uint4 a = ld_nc_v4(row + i);
    return make_uint4(pack_keys(a.x), pack_keys(a.y), pack_keys(a.z), pack_keys(a.w));
  }
  uint32_t k[4] = {0, 0, 0, 0};
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (i + e < V) {
      const uint32_t u = *reinterpret_cast<const unsigned short*>(row + i + e);
      k[e / 2] |= (pack_keys(u) & 0xffffu) << (16 * (e & 1));
    }
  return make_uint4(k[0], k[1], k[2], k[3]);
}

// STAGED: this CTA's part of the row stays in shared memory (as keys; a thread reads back only what it wrote); otherwise the row
// is too long for that and is read again, from L2, in every pass.
template <bool STAGED>
__global__ void __launch_bounds__(kSampleThreads, 2)
sample_kernel(int32_t* __restrict__ out, const bf16* __restrict__ logits, int V, int ld,
              const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ exp_noise,
              const uint64_t* __restrict__ seeds, uint64_t step) {
  __shared__ SampleShared sh;
  extern __shared__ uint4 held[];
  cluster_arrive_relaxed();                                  // see the wait below
  pdl_launch_dependents();
  pdl_wait();
  const int nc = (int)cluster_nctarank(), b = blockIdx.x / nc, tid = threadIdx.x;
  const bf16* row = logits + (int64_t)b * ld;
  const bool aligned = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  const float temp = temperature ? temperature[b] : 0.f;
  const bool greedy = temp < 1e-5f;
  const float inv_t = greedy ? 1.f : 1.f / temp;
  const int pieces = (V + 7) / 8, stride = nc * kSampleThreads, first = (int)cluster_ctarank() * kSampleThreads + tid;
  int phase = 0;

  if constexpr (STAGED) {
    // four loads in flight per thread
    int n = 0;
    for (int v8 = first; v8 < pieces; v8 += 4 * stride) {
      uint4 a[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) a[j] = v8 + j * stride < pieces ? load_keys(row, v8 + j * stride, V, aligned) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v8 + j * stride < pieces) held[(n + j) * kSampleThreads + tid] = a[j];
      n += 4;
    }
  }
  // f(key, index) for this thread's elements with lo <= key < lo + width.  The test of 32 elements makes a mask and only its set
  // bits are visited, so a pass over the few elements that still matter costs the test and little else.
  auto scan = [&](uint32_t lo, uint32_t width, auto&& f) {
    int n = tid;
#pragma unroll 1
    for (int v8 = first; v8 < pieces; v8 += 4 * stride, n += 4 * kSampleThreads) {
      uint32_t mask = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v8 + j * stride < pieces) {
          uint4 a;
          if constexpr (STAGED) a = held[n + j * kSampleThreads]; else a = load_keys(row, v8 + j * stride, V, aligned);
          const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (((e & 1) ? w[e / 2] >> 16 : w[e / 2] & 0xffffu) - lo < width) mask |= 1u << (8 * j + e);
        }
      while (mask) {
        const int s = __ffs(mask) - 1, j = s >> 3, e = s & 7, i = (v8 + j * stride) * 8 + e;
        mask &= mask - 1;
        uint32_t key;
        if constexpr (STAGED) key = reinterpret_cast<const unsigned short*>(held + n + j * kSampleThreads)[e];
        else key = pack_keys(*reinterpret_cast<const unsigned short*>(row + i)) & 0xffffu;
        f(key, i);
      }
    }
  };

  float best = -INFINITY;
  int bi = 0x7fffffff;
  auto offer = [&](float score, int i) { if (score > best || (score == best && i < bi)) { best = score; bi = i; } };
  constexpr uint32_t kTop = 0x8000u | kInfBits;                // the key of +inf; NaN lies above
  // this thread's largest key, with NaN and without
  int top[2] = {0, 0};
  int at = 0;
  {
    int n = tid;
#pragma unroll 1
    for (int v8 = first; v8 < pieces; v8 += stride, n += kSampleThreads) {
      uint4 a;
      if constexpr (STAGED) a = held[n]; else a = load_keys(row, v8, V, aligned);
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        int key = (int)((e & 1) ? w[e / 2] >> 16 : w[e / 2] & 0xffffu);
        if (greedy && key == 0x7fff) key = 0x8000;             // the two zeros are equal values
        if (key <= (int)kTop && key > top[0]) { top[0] = key; at = v8 * 8 + e; }
        top[1] = max(top[1], key);
      }
    }
  }
  cluster_wait();                                              // the peers run: their shared memory may be written
  if (greedy) {
    if (top[0]) offer(key_value(top[0]), at);                  // the first of equal keys
  } else {
    const int mine = top[1];
    cluster_reduce(top, sh, phase, MaxOp());
    const uint32_t mk = (uint32_t)top[0];
    const float m = mk ? key_value(mk) * inv_t : -INFINITY;    // max of x = logit / T: x grows with the key
    uint32_t cut = 1;                                          // keys from here on are kept
    auto lower_equal = [&]() {                                 // logits whose quotients are equal stay together
      const uint32_t t = fkey(key_value(cut) * inv_t);
      while (cut > 1 && fkey(key_value(cut - 1) * inv_t) >= t) --cut;
    };
    const int k = top_k ? top_k[b] : 0;
    if (k > 0 && k < V) {
      // the k-th largest key: largest v with count(key >= v) >= k, by cutting [lo, hi) in eight
      auto kth = [&](uint32_t lo, auto&& count) {
        uint32_t hi = (uint32_t)top[1] + 1;
        int want = k;
        while (hi - lo > 1) {
          const uint32_t w = (hi - lo + 7) / 8;
          int c[7] = {0, 0, 0, 0, 0, 0, 0};                    // elements at or above lo + w, lo + 2 w, ...
          count(lo, hi, w, c);
          cluster_reduce(c, sh, phase, AddOp());
          // counts are of [lo + j w, hi); those at or above hi were taken off `want` before
          int d = 7;
          while (d > 0 && c[d - 1] < want) --d;
          if (d < 7) want -= c[d];
          lo += (uint32_t)d * w;
          hi = min(hi, lo + w);
        }
        return lo;
      };
      // a thread's largest key stands for the thread: the k-th largest of those bounds the k-th largest of all from below
      uint32_t bound = 1;
      if (k <= stride / 4)
        bound = kth(1, [&](uint32_t lo, uint32_t hi, uint32_t w, int (&c)[7]) {
          if ((uint32_t)mine < hi) {
#pragma unroll
            for (int j = 0; j < 7; ++j) c[j] = (uint32_t)mine >= lo + (j + 1) * w;
          }
        });
      cut = kth(bound, [&](uint32_t lo, uint32_t hi, uint32_t w, int (&c)[7]) {
        scan(lo, hi - lo, [&](uint32_t key, int) {
#pragma unroll
          for (int j = 0; j < 7; ++j) c[j] += key >= lo + (j + 1) * w;
        });
      });
      lower_equal();
    }
    const float p = top_p ? top_p[b] : 1.f;
    if (p < 1.f) {
      // smallest key v with mass(key <= v) > (1-p) Z over the top-k survivors (ascending cumsum <= 1-p is dropped); a NaN among
      // the survivors leaves the largest logit alone
      // The interval [lo, hi) is cut at three keys per step: first at equal steps of the value (so that each step leaves about a
      // quarter of the logits in question), after four steps at equal steps of the key (so that it ends).
      uint32_t lo = min(cut, mk), hi = mk + 1;
      float below = 0.f, target = 0.f;
      if ((uint32_t)top[1] > kTop) lo = mk;
      const float vmax = key_value(mk), spread = 6.f / inv_t;
      float v0 = vmax - 4.f * spread, dv = spread;
#pragma unroll 1
      for (int it = 0; hi - lo > 1; ++it) {
        uint32_t cutat[3];
        const uint32_t w = (hi - lo + 3) / 4;
        uint32_t prev = lo;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float v = v0 + (j + 1) * dv;
          uint32_t c = it < 4 && fabsf(v) < 3e38f ? value_key(v) : lo + (j + 1) * w;
          c = min(max(c, prev + 1), hi);
          cutat[j] = prev = c;
        }
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        scan(lo, hi - lo, [&](uint32_t key, int) {
          const float e = expf(__fmul_rn(key_value(key), inv_t) - m);
          const int d = (key >= cutat[0]) + (key >= cutat[1]) + (key >= cutat[2]);
#pragma unroll
          for (int j = 0; j < 4; ++j) c[j] += d == j ? e : 0.f;
        });
        cluster_reduce(c, sh, phase, AddOp());
        if (it == 0) target = (1.f - p) * ((c[0] + c[1]) + (c[2] + c[3]));
        int d = 0;
        for (; d < 3 && cutat[d] < hi; ++d) {
          if (below + c[d] > target) break;
          below += c[d];
        }
        if (it == 0 && d == 0) it = 4;                         // far below the largest: by keys from here on
        if (d < 3) hi = cutat[d];
        if (d > 0) lo = cutat[d - 1];
        v0 += d * dv;
        dv *= 0.25f;
      }
      cut = max(cut, lo);
      lower_equal();
    }
    // argmax of exp(x - max) / q over the kept set; the maximum is always kept
    cut = min(cut, max(mk, 1u));
    const uint64_t seed = seeds ? seeds[b] : 0;
    scan(cut, 0x10000u - cut, [&](uint32_t key, int i) {
      const float q = exp_noise ? exp_noise[(int64_t)b * V + i] : -logf(philox_uniform(seed, step, (uint32_t)i));
      offer(expf(__fmul_rn(key_value(key), inv_t) - m) / q, i);
    });
  }
  const int lane = tid & 31, wid = tid >> 5;
  auto warp_best = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
  };
  warp_best();
  if (lane == 0) { sh.warp[0][wid] = __float_as_uint(best); sh.warp[1][wid] = (uint32_t)bi; }
  __syncthreads();
  if (wid == 0) {
    best = __uint_as_float(sh.warp[0][lane % kSampleWarps]);
    bi = (int)sh.warp[1][lane % kSampleWarps];
    warp_best();
    if (lane == 0) {
      st_cluster(&sh.all[phase & 1][cluster_ctarank()][0], 0, __float_as_uint(best));
      st_cluster(&sh.all[phase & 1][cluster_ctarank()][1], 0, (uint32_t)bi);
    }
  }
  cluster_arrive(); cluster_wait();
  if (cluster_ctarank() == 0 && tid == 0) {
    best = -INFINITY; bi = 0x7fffffff;
    for (int r = 0; r < nc; ++r) {
      const float ov = __uint_as_float(sh.all[phase & 1][r][0]);
      const int oi = (int)sh.all[phase & 1][r][1];
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    out[b] = bi == 0x7fffffff ? 0 : bi;
  }
}

}  // namespace KGE_ELT_NS
}  // namespace kge

using namespace kge;

#ifndef KGE_HALF
extern "C" int64_t kge_sample_workspace_bytes(int B, int V) {
  (void)B; (void)V;
  return 0;   // thresholds are found in shared memory; kept in the ABI for a future sort path
}

#endif

extern "C" int KGE_API(kge_sample)(int32_t* out_ids, const void* logits, int B, int V, int ld,
                          const float* temperature, const int32_t* top_k, const float* top_p,
                          const float* exp_noise, const uint64_t* seeds, uint64_t step, void* workspace,
                          int64_t workspace_bytes, void* stream) {
  (void)workspace; (void)workspace_bytes;
  KGE_REQUIRE(out_ids && logits && V > 0 && ld >= V, "kge_sample: bad arguments");
  if (B <= 0) return 0;
  // CTAs per row: enough that a thread has about 32 elements, and more while all rows together leave SMs idle (two CTAs fit on
  // one).  The latter at vocabulary 50272, us with and without: 32 rows of mixed settings 35.3 and 41.5, 1 row unfiltered 12.1
  // and 17.9; 64 rows (the rule leaves 4 CTAs) 46.0 and 45.7.
  const int64_t per = (int64_t)kSampleThreads * 32;
  int nc = 1;
  while (nc < kMaxCluster && nc * per < V) nc *= 2;
  while (nc < kMaxCluster && (int64_t)B * nc * 2 <= 2 * 148 && nc * (int64_t)kSampleThreads * 8 < V) nc *= 2;
  const int64_t trips = ((int64_t)(V + 7) / 8 + (int64_t)nc * kSampleThreads - 1) / ((int64_t)nc * kSampleThreads);
  const bool staged = trips * kSampleThreads * 16 <= 192 * 1024;
  const size_t smem = staged ? (size_t)(trips * kSampleThreads * 16) : 0;
  auto kern = staged ? sample_kernel<true> : sample_kernel<false>;
  // 48 KB of static and dynamic shared memory together go without the attribute (rows of 163841 to 196608 have 48 KB dynamic)
  if (smem + sizeof(SampleShared) > 48 * 1024) KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 192 * 1024));
  prefer_max_shared(kern);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)B * nc); cfg.blockDim = dim3(kSampleThreads); cfg.dynamicSmemBytes = smem; cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nc; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl_for_this_launch() ? 2 : 1;
  KGE_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, out_ids, (const bf16*)logits, V, ld, temperature, top_k, top_p, exp_noise, seeds, step));
  return 0;
}
