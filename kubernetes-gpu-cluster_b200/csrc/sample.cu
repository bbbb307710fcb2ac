// Temperature / top-k / top-p sampling, no sort.  A row belongs to a thread-block cluster; its CTAs hold the row's 16-bit
// logits in shared memory (as order-preserving integers) from one read of HBM / L2 on.  A 16-bit logit has few different values,
// so both thresholds come from ONE pass that counts them: 8192 counters in shared memory for the keys from the largest down
// (the tiny values around zero share one), each CTA then adds up a slice of them over its peers.
//   top-k   the largest key with k or more elements from it on: a scan of the counters;
//   top-p   the smallest key whose mass from below exceeds 1 - p: a scan of count * exp(value), one exponential per value that
//           occurs and not per element, over what lies below the counters (fp32, summed in a fixed order).
//           A threshold below the counted keys is looked for in the next 8192 (wide spreads in float16; never seen otherwise);
//   draw    the Gumbel-max form the reference uses, argmax(p_i / q_i) with q ~ Exp(1), over the kept set: each warp lists its kept
//           elements first and shares them out; q = -log u >= 1 - u tells without the logarithm that most cannot win.
// What bounds it: instruction issue of Philox (ten rounds per kept element) for flat rows, the chain of cluster barriers for the others (about
// 1 us each: the start's and the last exchange's for greedy rows, a third for the maximum where a token is drawn, three more for a threshold,
// two for a second one that finds its keys counted); the one read of V * 2 bytes is about 2 us.
// 32 rows x 128256 normal logits (spread 2.5) on a B200, us, before (intervals of keys cut in eight or four by a pass over the elements
// and a cluster exchange each, 6 to 12 of them; every kept element's logarithm) and now: greedy 6.8 / 4.8, top-k 20 with top-p 0.8
// 42.1 / 22.4, top-p 0.95 59.3 / 25.4, unfiltered 36.4 / 32.2, those in turn 51.2 / 23.9; one row of 32000, top-p 19.3 / 11.8; 150
// rows of 2049, top-k and top-p 31.5 / 17.5.
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

__device__ __forceinline__ uint2 ld_cluster_v2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(const void* local, uint32_t rank, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(mapa_u32((uint32_t)__cvta_generic_to_shared(local), rank)), "r"(v) : "memory");
}

constexpr int kSampleWarps = kSampleThreads / 32;
constexpr int kMaxCluster = 8;
constexpr int kBins = 8192;               // counters: 32 KB, which leaves 192 KB for the longest row that is kept
constexpr uint32_t kTop = 0x8000u | kInfBits;                // the key of +inf; NaN lies above

// Keys as bins: values near zero share one bin, or they, most of the format's range and hardly ever more than a few logits, would lie
// between the positive and the negative ones.
#ifdef KGE_HALF
constexpr uint32_t kPos = 0x8000u | 0x2400u;                 // the key of 2^-6: eight binades are counted at a time
#else
constexpr uint32_t kPos = 0x8000u | 0x3a00u;                 // 2^-11: from 2^5 to -2^5 in one go
#endif
constexpr uint32_t kNeg = 0xffffu - kPos;                    // the key of their negative
constexpr uint32_t kTiny = kNeg + 1, kGap = kPos - (kTiny + 1);
// Where a bin's counter is: threads that walk 16 (8, 4) bins each would meet in two (four, eight) banks.  Pairs stay pairs.
__device__ __forceinline__ uint32_t slot_of(uint32_t bin) { return bin ^ ((bin >> 3) & 14u); }
__device__ __forceinline__ uint32_t bin_of(uint32_t key) { return key >= kPos ? key - kGap : min(key, kTiny); }

struct SampleShared {
  uint32_t warp[2][kSampleWarps];
  uint32_t all[2][kMaxCluster][8];       // what every CTA of the cluster contributed, two exchanges in flight
  uint32_t found[2];                     // a search's result: the bin, and the sum up to and with it
  uint32_t last;
};

struct AddOp { template <typename T> __device__ __forceinline__ T operator()(T a, T b) const { return a + b; } };
struct MaxOp { template <typename T> __device__ __forceinline__ T operator()(T a, T b) const { return b > a ? b : a; } };

// Combine N <= 2 values over the cluster; every thread gets the results, combined in the same order everywhere.
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

// STAGED: this CTA's part of the row stays in shared memory (as keys); otherwise the row is too long for that and is read again,
// from L2, in every pass.
template <bool STAGED>
__global__ void __launch_bounds__(kSampleThreads, 2)
sample_kernel(int32_t* __restrict__ out, const bf16* __restrict__ logits, int V, int ld,
              const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
              const float* __restrict__ top_p, const float* __restrict__ exp_noise,
              const uint64_t* __restrict__ seeds, uint64_t step) {
  __shared__ SampleShared sh;
  extern __shared__ uint4 dyn[];
  uint32_t* hist = reinterpret_cast<uint32_t*>(dyn);         // [kBins]; the draw's lists afterwards
  uint4* held = dyn + kBins / 4;
  cluster_arrive_relaxed();                                  // see the wait below
  pdl_launch_dependents();
  pdl_wait();
  const int nc = (int)cluster_nctarank(), rank = (int)cluster_ctarank(), b = blockIdx.x / nc, tid = threadIdx.x;
  const int lane = tid & 31, wid = tid >> 5;
  const bf16* row = logits + (int64_t)b * ld;
  const bool aligned = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  const float temp = temperature ? temperature[b] : 0.f;
  const bool greedy = temp < 1e-5f;
  const float inv_t = 1.f / temp;
  const int pieces = (V + 7) / 8, stride = nc * kSampleThreads, first = rank * kSampleThreads + tid;
  int phase = 0;

  // Greedy rows, by themselves: the first element of the largest key, NaN left out, the two zeros equal.  What counts for few logits is the
  // instructions, and that they lie together (in one path with the draw a row of 1000 took 2.98 us, of 4695 3.45; 2.35 and 2.75 so).
  if (greedy) {
    int key = 0, piece = 0x7fffffff, n = tid;
#pragma unroll 1
    for (int v8 = first; v8 < pieces; v8 += 4 * stride, n += 4 * kSampleThreads) {
      uint4 a[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) if (v8 + j * stride < pieces) a[j] = load_keys(row, v8 + j * stride, V, aligned);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v8 + j * stride < pieces) {
          const uint32_t two = __vmaxu2(__vmaxu2(a[j].x, a[j].y), __vmaxu2(a[j].z, a[j].w));
          int k = (int)max(two & 0xffffu, two >> 16);
          if (k > (int)kTop) {                                 // a NaN among the eight
            const uint32_t w[4] = {a[j].x, a[j].y, a[j].z, a[j].w};
            k = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int x = (int)((e & 1) ? w[e / 2] >> 16 : w[e / 2] & 0xffffu);
              if (x <= (int)kTop) k = max(k, x);
            }
          }
          if (k == 0x7fff) k = 0x8000;
          if (k > key) { key = k; piece = v8 + j * stride; }
          if constexpr (STAGED) held[n + j * kSampleThreads] = a[j];
        }
    }
    auto first_of_largest = [&](int& k, int& at) {
      const int best = __reduce_max_sync(0xffffffffu, k);
      at = __reduce_min_sync(0xffffffffu, k == best ? at : 0x7fffffff);
      k = best;
    };
    first_of_largest(key, piece);
    if (lane == 0) { sh.warp[0][wid] = (uint32_t)key; sh.warp[1][wid] = (uint32_t)piece; }
    cluster_wait();                                            // the peers run: their shared memory may be written
    __syncthreads();
    if (wid == 0) {
      key = (int)sh.warp[0][lane % kSampleWarps];
      piece = (int)sh.warp[1][lane % kSampleWarps];
      first_of_largest(key, piece);
      int at = 0x7fffffff;
      if (key > 0) {                                           // which of the piece's eight
        uint32_t x = 0;
        const int i = piece * 8 + (lane & 7);
        if constexpr (STAGED) x = reinterpret_cast<const unsigned short*>(held + (piece & (kSampleThreads - 1)) + piece / stride * kSampleThreads)[lane & 7];
        else if (i < V) x = pack_keys(*reinterpret_cast<const unsigned short*>(row + i)) & 0xffffu;
        at = __reduce_min_sync(0xffffffffu, (int)x == key || (x == 0x7fffu && key == 0x8000) ? i : 0x7fffffff);
      }
      if (lane == 0) {
        st_cluster(&sh.all[0][rank][0], 0, (uint32_t)key);
        st_cluster(&sh.all[0][rank][1], 0, (uint32_t)at);
      }
    }
    cluster_arrive(); cluster_wait();
    if (rank == 0 && wid == 0) {
      key = lane < nc ? (int)sh.all[0][lane & (kMaxCluster - 1)][0] : 0;
      int at = lane < nc ? (int)sh.all[0][lane & (kMaxCluster - 1)][1] : 0x7fffffff;
      first_of_largest(key, at);
      if (lane == 0) out[b] = at == 0x7fffffff ? 0 : at;
    }
    return;
  }

  // this thread's largest key, with NaN: of even and odd elements side by side
  uint32_t both = 0;
  {
    // four loads in flight per thread
    int n = tid;
#pragma unroll 1
    for (int v8 = first; v8 < pieces; v8 += 4 * stride, n += 4 * kSampleThreads) {
      uint4 a[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) a[j] = v8 + j * stride < pieces ? load_keys(row, v8 + j * stride, V, aligned) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        both = __vmaxu2(both, __vmaxu2(__vmaxu2(a[j].x, a[j].y), __vmaxu2(a[j].z, a[j].w)));
        if constexpr (STAGED)
          if (v8 + j * stride < pieces) held[n + j * kSampleThreads] = a[j];
      }
    }
  }
  // f(packed keys of 8 elements, index of the first) for this thread's elements
  auto each8 = [&](auto&& f) {
    int n = tid;
#pragma unroll 1
    for (int v8 = first; v8 < pieces; v8 += stride, n += kSampleThreads) {
      uint4 a;
      if constexpr (STAGED) a = held[n]; else a = load_keys(row, v8, V, aligned);
      f(a, v8 * 8);
    }
  };

  float best = -INFINITY, floor = 0.f;
  int bi = 0x7fffffff;
  auto offer = [&](float score, int i) { if (score > best || (score == best && i < bi)) { best = score; bi = i; } };
  int top[2];                                                  // the largest key without NaN, and with
  top[1] = (int)max(both & 0xffffu, both >> 16);
  top[0] = top[1];
  if (top[1] > (int)kTop) {                                    // a NaN here
    top[0] = 0;
    each8([&](uint4 a, int) {
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int key = (int)((e & 1) ? w[e / 2] >> 16 : w[e / 2] & 0xffffu);
        if (key <= (int)kTop) top[0] = max(top[0], key);
      }
    });
  }
  float m = 0.f;
  uint32_t low = 0, from = 0;                                  // the kept keys, and those of them that are drawn from
  auto weight = [&](uint32_t key) { return expf(__fmul_rn(key_value(key), inv_t) - m); };
  cluster_wait();                                              // the peers run: their shared memory may be written
  cluster_reduce(top, sh, phase, MaxOp());
  const uint32_t mk = (uint32_t)top[0];
  m = mk ? key_value(mk) * inv_t : -INFINITY;    // max of x = logit / T: x grows with the key
  uint32_t cut = 1;                                          // keys from here on are kept
  auto lower_equal = [&]() {                                 // logits whose quotients are equal stay together
    const uint32_t t = fkey(key_value(cut) * inv_t);
    while (cut > 1 && fkey(key_value(cut - 1) * inv_t) >= t) --cut;
  };
  const int k = top_k ? top_k[b] : 0;
  const float p = top_p ? top_p[b] : 1.f;

  // Counts of the bins [base, base + width) into `hist`; `tiny` is the weight of the shared bin and `rest` that of the bins below
  // base, over the cluster, of keys from `low` on.  `raw`: bins are keys, inside the shared bin.
  float rest = 0.f, tiny = 0.f;
  auto count = [&](uint32_t base, uint32_t width, bool raw, uint32_t low, bool weights) {
    for (int i = tid; i < kBins / 4; i += kSampleThreads) dyn[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    float s[2] = {0.f, 0.f};
    uint32_t small = 0;                                      // elements of the shared bin: counted here, there may be many
    each8([&](uint4 a, int) {
      const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t key = (e & 1) ? w[e / 2] >> 16 : w[e / 2] & 0xffffu, c = raw ? key : bin_of(key);
        const bool shared = !raw && c == kTiny;
        if (c - base < width && !shared) atomicAdd(hist + slot_of(c - base), 1u);
        if (shared || c < base) {
          small += shared;
          if (weights && key >= low) {
            const float x = weight(key);
            s[0] += c < base ? x : 0.f;
            s[1] += shared ? x : 0.f;
          }
        }
      }
    });
    if (!raw && kTiny - base < width && small) atomicAdd(hist + slot_of(kTiny - base), small);
    cluster_reduce(s, sh, phase, AddOp());                   // the counters are complete behind it
    rest = s[0];
    tiny = s[1];
    // Each CTA adds up a slice, a thread `per` bins in a row.  Nobody else reads that slice of this CTA's counters.
    const int per = kBins / stride;
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(hist);
    for (int j = 0; j < per && nc > 1; j += 2) {
      const uint32_t at = slot_of((uint32_t)(first * per + j));
      uint32_t x = 0, y = 0;
#pragma unroll
      for (int r = 0; r < kMaxCluster; ++r)
        if (r < nc) {
          const uint2 v = ld_cluster_v2(mapa_u32(mine + at * 4, (uint32_t)r));
          x += v.x;
          y += v.y;
        }
      hist[at] = x;
      hist[at + 1] = y;
    }
  };
  // The first bin whose sum from below exceeds want(sum of all slices), by value(bin, count): the same everywhere.  kBins: it lies
  // below the counted ones; kBins + 1: there is none.  `upto` is the sum up to and with the bin.
  auto find = [&](auto value, auto want_of, auto& upto) -> uint32_t {
    using T = typename std::remove_reference<decltype(upto)>::type;
    const int per = kBins / stride;
    T sum = 0;
    for (int j = 0; j < per; ++j) sum += value((uint32_t)(first * per + j), hist[slot_of((uint32_t)(first * per + j))]);
    T incl = sum;                                            // over the threads of the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    T start = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) start = 0;
    T* warp = reinterpret_cast<T*>(sh.warp[0]);
    if (lane == 31) warp[wid] = incl;
    if (tid == 0) sh.last = 0;
    __syncthreads();
    T before = 0, all = 0;
    for (int w = 0; w < kSampleWarps; ++w) {
      if (w == wid) before = all;
      all += warp[w];
    }
    if (tid < nc) st_cluster(&sh.all[phase & 1][rank][0], (uint32_t)tid, *reinterpret_cast<uint32_t*>(&all));
    cluster_arrive(); cluster_wait();
    T total = 0, below = 0;
    for (int r = 0; r < nc; ++r) total += *reinterpret_cast<T*>(&sh.all[phase & 1][r][0]);
    const T want = want_of(total);
    total = 0;
    int owner = -1;
    for (int r = 0; r < nc; ++r) {
      const T next = total + *reinterpret_cast<T*>(&sh.all[phase & 1][r][0]);
      if (owner < 0 && next > want) { owner = r; below = total; }
      total = next;
    }
    ++phase;
    if (want < 0) return kBins;
    if (owner < 0) return kBins + 1;
    if (owner == rank) {
      // the last thread that starts at or below `want` and adds something: sums of fp32 differ by their order, so no thread's
      // end is compared with the next one's start
      start = below + (before + start);
      if (sum > 0 && start <= want) atomicMax(&sh.last, (uint32_t)tid);
      __syncthreads();
      if (tid == (int)sh.last) {
        T run = start;
        uint32_t at = kBins + 1;
        for (int j = 0; j < per && !(run > want); ++j)
          if (const uint32_t n = hist[slot_of((uint32_t)(first * per + j))]) {
            at = (uint32_t)(first * per + j);
            run += value(at, n);
          }
        for (int r = 0; r < nc; ++r) {
          st_cluster(&sh.found[0], (uint32_t)r, at);
          st_cluster(&sh.found[1], (uint32_t)r, *reinterpret_cast<uint32_t*>(&run));
        }
      }
    }
    cluster_arrive(); cluster_wait();
    upto = *reinterpret_cast<T*>(&sh.found[1]);
    return sh.found[0];
  };
  // mass: the smallest key whose weight from below exceeds (1 - p) of all, of the keys from `low` on; else the k-th largest key.
  // counted: the counters hold the first bins already, and `low` lies among them, above the shared one.
  auto search = [&](int mass, uint32_t largest, uint32_t low, bool counted) -> uint32_t {
    uint32_t hi = bin_of(largest) + 1, lowest = 1;
    bool raw = false;
    int above = 0, ends = 0;
    float goal = -1.f;
    for (;;) {
      const uint32_t base = hi - lowest > kBins ? hi - kBins : lowest;
      if (!counted) count(base, hi - base, raw, low, mass); else rest = tiny = 0.f;
      counted = false;
      uint32_t at;
      int all = 0;
      if (mass) {
        float upto;
        at = find([&](uint32_t i, uint32_t n) -> float {
          const uint32_t c = base + i, key = raw || c <= kNeg ? c : c + kGap;
          if (n == 0) return 0.f;
          if (!raw && c == kTiny) return tiny;
          return key >= low ? (float)n * weight(key) : 0.f;
        }, [&](float total) {
          if (goal == -1.f) goal = (1.f - p) * (rest + total);
          return goal - rest;
        }, upto);
      } else {
        at = find([](uint32_t, uint32_t n) { return (int)n; }, [&](int total) { all = total; return above + total - k; }, ends);
      }
      if (at == kBins + 1) return largest;
      if (at == kBins) {
        if (base == lowest) return lowest;                   // by rounding only
        above += all;
        hi = base;
        continue;
      }
      at += base;
      if (raw || at != kTiny) return raw || at <= kNeg ? at : at + kGap;
      above += all - ends;
      raw = true;
      hi = kPos;
      lowest = kTiny;
    }
  };
  bool counted = false;
#pragma unroll 1
  for (int mass = 0; mass < 2; ++mass) {
    if (mass ? !(p < 1.f) : !(k > 0 && k < V)) continue;
    if (mass && top[1] > (int)kTop) { cut = max(cut, mk); continue; }       // a NaN leaves the largest logit alone
    const uint32_t key = search(mass, (uint32_t)(mass ? mk : top[1]), cut, counted);
    const uint32_t hi = bin_of((uint32_t)top[1]) + 1, at = bin_of(key);
    cut = max(cut, key);
    lower_equal();
    // whether the counters are the first ones still, and what the threshold of the mass needs is in them
    counted = at > kTiny && at + kBins >= hi && bin_of(cut) > kTiny && bin_of(cut) + kBins >= hi;
  }
  // argmax of exp(x - max) / q over the kept set; the maximum is always kept
  cut = min(cut, max(mk, 1u));
  // The largest score is W / Exp(1), W >= 1 the kept weights' sum: below `floor` with a probability of e^-16.7, and then the draw
  // is repeated without it.  What cannot reach it, or the best score of the warp so far, is left out before its logarithm.
  floor = 0.06f;
  low = from = cut;
  if (exp_noise) floor = 0.f;
  else {
    const float v = (m - 19.6f) * temp;                      // q >= 2^-24.1: a weight below e^-19.45 cannot reach 0.06
    if (fabsf(v) < 3e4f && fabsf(m) < 1e5f) from = min(max(cut, value_key(v) - 1), max(mk, 1u));
  }
  const uint64_t seed = seeds ? seeds[b] : 0;
  uint16_t* list = reinterpret_cast<uint16_t*>(hist) + wid * 1024;
  auto draw = [&]() {
    float reach = floor;
    int n = tid;
#pragma unroll 1
    for (int v8 = first; v8 - lane < pieces; v8 += 4 * stride, n += 4 * kSampleThreads) {
      uint32_t mask = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v8 + j * stride < pieces) {
          uint4 a;
          if constexpr (STAGED) a = held[n + j * kSampleThreads]; else a = load_keys(row, v8 + j * stride, V, aligned);
          const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (((e & 1) ? w[e / 2] >> 16 : w[e / 2] & 0xffffu) >= from) mask |= 1u << (8 * j + e);
        }
      // where all lanes keep the same first pieces whole (nothing is cut, mostly), the lists need not be written
      const bool alike = __all_sync(0xffffffffu, mask == __shfl_sync(0xffffffffu, mask, 0) && (mask & (mask + 1)) == 0);
      int total = 32 * __popc(mask);
      if (!alike) {
        int upto = __popc(mask);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += v;
        }
        total = __shfl_sync(0xffffffffu, upto, 31);
        __syncwarp();                                          // the list was read
        for (uint16_t* to = list + upto - __popc(mask); mask; mask &= mask - 1) *to++ = (uint16_t)(lane << 5 | (__ffs(mask) - 1));
        __syncwarp();
      }
      // Philox is a chain of ten rounds: two elements a turn
#pragma unroll 1
      for (int t = lane; t - lane < total; t += 64) {
        uint32_t key[2];
        int at[2];
        float u[2];
        bool may[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          may[h] = t + 32 * h < total;
          const int s = alike || !may[h] ? lane << 5 | ((t >> 5) + h & 31) : list[t + 32 * h];
          const int l = (s >> 5) - lane, j = (s >> 3) & 3, e = s & 7;
          at[h] = (v8 + l + j * stride) * 8 + e;
          key[h] = 0;
          if (may[h]) {
            if constexpr (STAGED) key[h] = reinterpret_cast<const unsigned short*>(held + n + l + j * kSampleThreads)[e];
            else key[h] = pack_keys(*reinterpret_cast<const unsigned short*>(row + at[h])) & 0xffffu;
          }
        }
        if (exp_noise) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (may[h]) offer(weight(key[h]) / exp_noise[(int64_t)b * V + at[h]], at[h]);
          continue;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) u[h] = philox_uniform(seed, step, (uint32_t)at[h]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float about;                                         // weight(key) within 2^-12
          asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(about) : "f"((__fmul_rn(key_value(key[h]), inv_t) - m) * 1.44269504f));
          may[h] = may[h] && !(about < reach * (1.f - u[h]) * 0.998f);
        }
        if (__any_sync(0xffffffffu, may[0] || may[1])) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (may[h]) offer(weight(key[h]) / -logf(u[h]), at[h]);
          reach = fmaxf(reach, warp_max(best));
        }
      }
    }
  };
  auto warp_best = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
  };
#pragma unroll 1
  for (;;) {
    draw();
    // the best of the cluster, of equal ones the first: known to every CTA
    warp_best();
    if (lane == 0) { sh.warp[0][wid] = __float_as_uint(best); sh.warp[1][wid] = (uint32_t)bi; }
    __syncthreads();
    if (wid == 0) {
      best = __uint_as_float(sh.warp[0][lane % kSampleWarps]);
      bi = (int)sh.warp[1][lane % kSampleWarps];
      warp_best();
      if (lane < nc) {
        st_cluster(&sh.all[phase & 1][rank][0], (uint32_t)lane, __float_as_uint(best));
        st_cluster(&sh.all[phase & 1][rank][1], (uint32_t)lane, (uint32_t)bi);
      }
    }
    cluster_arrive(); cluster_wait();
    best = lane < nc ? __uint_as_float(sh.all[phase & 1][lane & (kMaxCluster - 1)][0]) : -INFINITY;
    bi = lane < nc ? (int)sh.all[phase & 1][lane & (kMaxCluster - 1)][1] : 0x7fffffff;
    warp_best();
    ++phase;
    if (best >= floor || floor == 0.f) break;
    floor = 0.f;
    from = low;
    best = -INFINITY; bi = 0x7fffffff;
  }
  if (rank == 0 && tid == 0) out[b] = bi == 0x7fffffff ? 0 : bi;
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
  const size_t smem = kBins * 4 + (staged ? (size_t)(trips * kSampleThreads * 16) : 0);
  auto kern = staged ? sample_kernel<true> : sample_kernel<false>;
  // 48 KB of static and dynamic shared memory together go without the attribute
  if (smem + sizeof(SampleShared) > 48 * 1024) KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 192 * 1024 + kBins * 4));
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
