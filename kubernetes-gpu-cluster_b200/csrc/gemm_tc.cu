// Dense projection  y[T,N] = act(x[T,K] * w[N,K]^T + bias)  on the 5th-gen tensor cores.
//
// Weight-stationary orientation ("swap-AB"): the 128-row MMA M dimension runs over WEIGHT rows
// (N is always large: 768..128256) and the MMA N dimension (16..256) over TOKENS, so a decode
// step with T = 16..256 tokens wastes no tensor-core rows and streams every weight byte exactly
// once.  D[weight row, token] lives in TMEM (fp32); the epilogue reads it back with tcgen05.ld as
// MMA fragments, adds the bias of their rows, applies the activation, rounds once to 16 bits, and
// stmatrix turns the fragments so that a lane stores 16 bytes of an output row.
// Which kernel: up to 16 tokens, by size, gemm_rows.cuh (weights streamed without staging tiles); 33
// to 64 tokens where 128-row tiles would be split in two, gemm_wide_kernel; above 64 CTA pairs with a
// token tile of 32 to 256 (plan_pairs); single-CTA tiles elsewhere.
//
// Persistent, warp-specialised: warp 0 = TMA producer (cp.async.bulk.tensor, 128B swizzle),
// warp 1 = tcgen05.mma issuer (one elected lane), warp 2 = TMEM allocator, warps 4-7 = epilogue.
// smem ring of STAGES {W tile 128x64, X tile TOKNx64}; two TMEM accumulator stages so the
// epilogue of tile i overlaps the main loop of tile i+1.
// Split-K (decode, when N/128 tiles cannot fill 148 SMs): the S CTAs of a thread-block CLUSTER
// share one output tile and each take 1/S of K.  Their fp32 partial accumulators are exchanged
// through distributed shared memory (st.shared::cluster): CTA r receives column slice r of every
// peer, sums the S partials in rank order (deterministic), adds bias, rounds once and stores.
// No global scratch, no atomics, no serial tail; the cluster guarantees co-scheduling.
// Stream-K through a workspace (WS; decode-sized projections when the caller provides scratch): the (tile, k-block) units
// of the whole problem are laid end to end and cut into one contiguous share per CTA, one CTA per SM - every SM streams
// exactly 1/148 of the weights through ONE uninterrupted TMA ring, whatever the tile count (48 tiles x split 2 used 96 SMs,
// 224 tiles used 112).  A CTA's share covers at most one partial tile at its start and one at its end: those fp32 partials
// go to the workspace (they stay in L2) and the CTA that arrives LAST on the tile's counter sums the tile's partials in
// k order (deterministic), applies bias / activation / SiLU-gate, rounds once and stores; whole tiles in between take the
// ordinary epilogue.  The accumulators are double-buffered in TMEM, so all of this overlaps the next segment's main loop.
//
// Roofline: decode T<=256 -> HBM, algorithmic bytes = N*K*2 (weights) + T*(K+N)*2;
//           prefill        -> tensor, 2*T*N*K flop.
#include <cuda.h>
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "kge.h"
#include "norm_gemm.h"

namespace kge {
inline namespace KGE_ELT_NS {

constexpr int BLK_M = 128;   // weight rows per tile (UMMA M)
constexpr int BLK_K = 64;    // 64 bf16 = 128 B = one swizzle row
constexpr int UMMA_K = 16;
constexpr int kGemmThreads = 256;
constexpr int kPairSub = 2;     // k-blocks per stage of the pair kernel: half the barriers (64-token tiles 0.30 -> 0.25 us a k-block)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// The same loads with an L2 eviction-priority hint (knob gemm_l2_hints): weights are read once per launch (evict_first),
// the activation tile is re-read by every CTA (evict_last), so the prefill GEMM stops re-fetching X from HBM behind its
// own output stream (without it 2.42 GB of DRAM traffic for 0.77 GB of algorithmic bytes on the gate_up shape).
__device__ __forceinline__ uint64_t l2_policy(bool keep) {
  uint64_t pol;
  if (keep) asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
  else asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, uint64_t pol) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "l"(pol) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
               ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
  tmem_wait_ld(r);
}

// 16 TMEM lanes x 8 G columns as MMA accumulator fragments: register 4 k + i holds lane (l / 4) + 8 (i / 2), column 8 k + 2 (l % 4) + i % 2.
// The caller waits (tmem_wait_ld).
template <int G>
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t (&r)[4 * G]) {
  static_assert(G == 2 || G == 4, "");
  if constexpr (G == 4)
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
  else
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void stsm_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// K-major, 128B-swizzled operand tile (rows of 128 B, 8-row atoms 1024 B apart).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;                    // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset between 8-row atoms
  d |= (uint64_t)1 << 46;                    // descriptor version (Blackwell)
  d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
  return d;
}

struct GemmParams {
  bf16* y;
  const bf16* bias;
  float* ws_part;            // WS: [tile][split][token column][128 rows] fp32 partial accumulators
  unsigned int* ws_count;    // WS: per-tile arrival counters (zero before the first launch; the reducing CTA resets its own)
  int T, N, K, act;
  int l2_hints;              // 1: weights evict_first, activations evict_last, output stored streaming
  int m_tiles, n_tiles, splits, kb_total, kb_per_split;
  int tokn = 0;              // PAIR: tokens per tile, a multiple of 32 up to 256
  unsigned long long* trace; // phase timestamps, 16 per CTA (tools/gemm_trace.py); null outside that tool
  int glu = 0;               // gated pair: 0 silu(gate) * up; 1 clamped: g = min(gate, limit), u = clamp(up, +-limit), g * sigmoid(alpha g) * (u + 1)
  float glu_alpha = 0.f, glu_limit = 0.f;
  // grouped rows (mixture of experts): token rows come in groups padded to multiples of 256, tile_group[i] names the weight
  // slice of rows [256 i, 256 (i + 1)) (negative: no rows, y is left alone), and slice g starts at weight row g * group_rows of the stacked weight tensor
  const int32_t* tile_group = nullptr;
  int group_rows = 0;
};

// epilogue activation of the plain projection: 0 none, 1 relu, 3 exact (erf) gelu; 2 marks the gated pair internally
__device__ __forceinline__ float apply_act(float v, int act) {
  if (act == 1) return fmaxf(v, 0.f);
  if (act == 3) return 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
  if (act == 4) { const float r = fmaxf(v, 0.f); return r * r; }
  return v;
}


// One %globaltimer stamp of this CTA's phase `slot` (see tools/gemm_trace.py for the slot list).
__device__ __forceinline__ void trace_stamp(const GemmParams& p, int slot) {
  if (p.trace) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t) :: "memory");
    p.trace[(size_t)blockIdx.x * 16 + slot] = t;
  }
}

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_f4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// exchange buffer of the split variant: [src rank][local column][128 rows] fp32
__host__ __device__ constexpr int xbuf_bytes(int tokn) { return (tokn + 8) * BLK_M * 4; }

// the gated pair of pre-activations that are rounded already
__device__ __forceinline__ float silu_gate_rounded(const GemmParams& p, float g, float u) {
  if (p.glu == 1) {                                      // clamped pair with a sigmoid gate: fp32 from the rounded pre-activations
    g = fminf(g, p.glu_limit);
    u = fminf(fmaxf(u, -p.glu_limit), p.glu_limit);
    return __fdividef(g, 1.0f + __expf(-p.glu_alpha * g)) * (u + 1.0f);
  }
  const float sg = rbf(__fdividef(g, 1.0f + __expf(-g))); // F.silu rounds to bf16 (fast exp/div: <= 2 ulp in fp32)
  return sg * u;                                          // caller rounds the product once
}

// GATED: the 128 MMA rows of a tile are 64 gate rows (TMEM lanes 0-63) and the matching 64 up rows
// (lanes 64-127) of a stacked [2f, K] weight; the epilogue emits silu(gate) * up for the 64
// outputs with vLLM's cast points (vllm:model_executor/layers/activation.py:137-141).
// n: the output column; with a bias ([gate | up] halves of p.N numbers each) it joins the accumulators before the rounding.
__device__ __forceinline__ float silu_gate_bf16(const GemmParams& p, float g_acc, float u_acc, int n) {
  if (p.bias && n < p.N) { g_acc += bf2f(p.bias[n]); u_acc += bf2f(p.bias[p.N + n]); }
  return silu_gate_rounded(p, rbf(g_acc), rbf(u_acc));   // the gate_up GEMM output is bf16
}

__device__ __forceinline__ void tma_load_2d_cg2_hint(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1, uint64_t pol) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
               ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1), "l"(pol) : "memory");
}
__device__ __forceinline__ void tma_load_2d_cg2(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tc_commit_cg2(uint32_t bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void tc_mma_bf16_cg2(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
               ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}

// PAIR (TOKN = 256 columns of TMEM per accumulator): cta_group::2.  The two CTAs of a cluster form one
// MMA tile of 256 weight rows x p.tokn tokens: each holds its own 128 weight rows (A) and HALF of the
// token tile (B, up to 128 tokens) in shared memory (32 KB per k-block instead of 48 KB: less L2->SM
// traffic and less shared-memory bandwidth; two k-blocks per stage, three stages), the leader CTA issues tcgen05.mma.cta_group::2 for both, accumulators land in each CTA's own TMEM.
// All TMA loads of a stage complete on the LEADER's full barrier; tcgen05.commit multicasts the
// "stage free" and "accumulator ready" arrivals to both CTAs; both epilogues release the accumulator
// on the leader's tmem_empty barrier.  The width of the token tile is a launch parameter (p.tokn): the host picks what leaves
// the last round of tiles fullest.
// PAIR && SPLIT: a cluster of S pairs shares one tile, each pair takes 1/S of K.  Once all of them are past their main loops the
// pipeline stages hold the exchange: pair o finishes the o-th share of the tile's 32-token groups, and every other pair sends it
// its fp32 accumulators of those, in the fragment order in which the epilogue reads TMEM (512-byte warp stores); the owner adds
// them in rank order.
template <int TOKN, int STAGES, bool SPLIT, bool GATED, bool PAIR = false, bool WS = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
               const GemmParams p) {
  static_assert(!(WS && (SPLIT || PAIR)), "one split scheme at a time");
  constexpr bool XSPLIT = SPLIT && !PAIR;               // K split over single CTAs, exchanged through a buffer of its own
  constexpr uint32_t A_BYTES = BLK_M * BLK_K * 2, B_BYTES = (PAIR ? 128 : TOKN) * BLK_K * 2;
  constexpr int SUB = PAIR ? kPairSub : 1;               // k-blocks per stage
  constexpr uint32_t STAGE_BYTES = SUB * (A_BYTES + B_BYTES);
  constexpr uint32_t TMEM_COLS = (2 * TOKN < 32) ? 32 : 2 * TOKN;
  const int tokn = PAIR ? p.tokn : TOKN;
  const uint32_t IDESC = (1u << 4) | KGE_IDESC_AB | ((uint32_t)(tokn >> 3) << 17) |
                         ((uint32_t)((PAIR ? 2 * BLK_M : BLK_M) >> 4) << 24);

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  // bars: full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  float* xbuf = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES + 2048);   // SPLIT: exchange buffer;
                                                                                // GATED && !SPLIT: gate / up hand-off, 8 KB
  constexpr int ROWS_OUT = GATED ? 64 : BLK_M;           // output columns produced per tile
  const uint32_t smem_base = smem_addr(smem);
  const uint32_t bar_base = smem_addr(bars);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };
  auto tempty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + 2 + s); };

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    trace_stamp(p, 0);
    if (p.trace) { uint32_t sm; asm volatile("mov.u32 %0, %%smid;" : "=r"(sm)); p.trace[(size_t)blockIdx.x * 16 + 15] = sm; }
  }
  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(tfull_bar(s), 1); mbar_init(tempty_bar(s), PAIR ? 8 : 4); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "n"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "n"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) trace_stamp(p, 1);
  if (PAIR) { cluster_arrive(); cluster_wait(); }   // peer barriers are initialised before any remote signal
  // TMEM is held: the next kernel may start arriving now (see attn_tc.cu for why not earlier)
  pdl_launch_dependents();
  if (warp != 0) pdl_wait();          // warp 0 (TMA producer) prefetches weights first, then waits

  // work decomposition: persistent round-robin over tiles, or (SPLIT) one tile per cluster with
  // the cluster rank selecting the K range
  const int S = SPLIT ? (int)cluster_nctarank() / (PAIR ? 2 : 1) : 1;
  const int crank = SPLIT ? (int)cluster_ctarank() / (PAIR ? 2 : 1) : 0;      // which share of K
  constexpr bool TWO = PAIR;
  const int mrank = TWO ? (int)cluster_ctarank() & 1 : 0;        // which tile of the weight-row pair
  const uint32_t leader = TWO ? cluster_ctarank() & ~1u : 0u;    // the pair's CTA that issues the MMAs
  const int total = (TWO ? (p.m_tiles + 1) / 2 : p.m_tiles) * p.n_tiles;
  const int w_first = SPLIT ? (int)blockIdx.x / (PAIR ? 2 * S : S) : TWO ? (int)blockIdx.x / 2 : (int)blockIdx.x;
  const int w_step = SPLIT ? (1 << 30) : TWO ? (int)gridDim.x / 2 : (int)gridDim.x;
  auto m_tile_of = [&](int w) { return TWO ? 2 * (w / p.n_tiles) + mrank : w / p.n_tiles; };
  // grouped rows: a tile beyond the last group has no work (every role reads the table after pdl_wait and skips alike)
  auto no_rows = [&](int w) { return p.tile_group != nullptr && p.tile_group[((w % p.n_tiles) * tokn) >> 8] < 0; };
  // PAIR: every TMA of a stage completes on the leader's full barrier
  auto lead_full = [&](int s) { return PAIR ? mapa_u32(full_bar(s), leader) : full_bar(s); };
  const int kb0f = crank * p.kb_per_split, kb1f = min(p.kb_total, kb0f + p.kb_per_split);
  const int cols_per = (TOKN + S - 1) / S;               // columns finished by each cluster rank
  // A CTA's work as a sequence of segments (tile w, k-blocks [kb0, kb1)).  Persistent / split variants: its tiles, each
  // with the same k range.  WS (stream-K): its contiguous share [u_begin, u_end) of the tiles * kb_total units.
  const int KB = p.kb_total;
  const int64_t U = (int64_t)total * KB;
  const int64_t u_begin = WS ? U * (int64_t)blockIdx.x / (int64_t)gridDim.x : 0;
  const int64_t u_end = WS ? U * ((int64_t)blockIdx.x + 1) / (int64_t)gridDim.x : 0;
  struct SegIter {
    int64_t cur, end;
    int step, KB, k0, k1;
    __device__ __forceinline__ bool next(int& w, int& kb0, int& kb1) {
      if (cur >= end) return false;
      if (WS) {
        w = (int)(cur / KB); kb0 = (int)(cur % KB);
        const int64_t left = end - cur;
        kb1 = (left < (int64_t)(KB - kb0)) ? kb0 + (int)left : KB;
        cur += kb1 - kb0;
      } else {
        w = (int)cur; kb0 = k0; kb1 = k1; cur += step;
      }
      return true;
    }
  };
  auto segments = [&]() { return WS ? SegIter{u_begin, u_end, 0, KB, 0, 0} : SegIter{(int64_t)w_first, (int64_t)total, w_step, KB, kb0f, kb1f}; };
  if (XSPLIT) cluster_arrive_relaxed();                  // phase A: every CTA of the cluster has started (nothing to publish: no release)

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0; uint32_t phase = 0;
      const bool hint = p.l2_hints != 0;
      const uint64_t pol_w = l2_policy(false), pol_x = l2_policy(true);
      auto load_a = [&](int st, int kb, int m_tile, int woff, int sub) {
        const uint32_t a_dst = smem_base + st * STAGE_BYTES + sub * (A_BYTES + B_BYTES);
        kb += sub;
        if (PAIR && hint) {
          if (GATED) {
            tma_load_2d_cg2_hint(a_dst, &tmap_w, lead_full(st), kb * BLK_K, woff + m_tile * 64, pol_w);
            tma_load_2d_cg2_hint(a_dst + 64 * BLK_K * 2, &tmap_w, lead_full(st), kb * BLK_K, woff + p.N + m_tile * 64, pol_w);
          } else {
            tma_load_2d_cg2_hint(a_dst, &tmap_w, lead_full(st), kb * BLK_K, woff + m_tile * BLK_M, pol_w);
          }
        } else if (PAIR) {
          if (GATED) {
            tma_load_2d_cg2(a_dst, &tmap_w, lead_full(st), kb * BLK_K, woff + m_tile * 64);
            tma_load_2d_cg2(a_dst + 64 * BLK_K * 2, &tmap_w, lead_full(st), kb * BLK_K, woff + p.N + m_tile * 64);
          } else {
            tma_load_2d_cg2(a_dst, &tmap_w, lead_full(st), kb * BLK_K, woff + m_tile * BLK_M);
          }
        } else if (hint) {
          if (GATED) {
            tma_load_2d_hint(a_dst, &tmap_w, full_bar(st), kb * BLK_K, woff + m_tile * 64, pol_w);
            tma_load_2d_hint(a_dst + 64 * BLK_K * 2, &tmap_w, full_bar(st), kb * BLK_K, woff + p.N + m_tile * 64, pol_w);
          } else {
            tma_load_2d_hint(a_dst, &tmap_w, full_bar(st), kb * BLK_K, woff + m_tile * BLK_M, pol_w);
          }
        } else if (GATED) {
          tma_load_2d(a_dst, &tmap_w, full_bar(st), kb * BLK_K, woff + m_tile * 64);                          // gate rows
          tma_load_2d(a_dst + 64 * BLK_K * 2, &tmap_w, full_bar(st), kb * BLK_K, woff + p.N + m_tile * 64);   // up rows
        } else {
          tma_load_2d(a_dst, &tmap_w, full_bar(st), kb * BLK_K, woff + m_tile * BLK_M);
        }
      };
      // the barrier that counts a stage's bytes: its own or, PAIR, the leader's for both CTAs
      auto expect = [&](int st, int subs) {
        if (!PAIR) mbar_expect_tx(full_bar(st), STAGE_BYTES);
        else if (mrank == 0) mbar_expect_tx(full_bar(st), subs * (2 * A_BYTES + (uint32_t)tokn * BLK_K * 2));
      };
      // Weights do not depend on the previous kernel: stream the first stages of W while it is
      // still running, then wait for its output (the activations) and add the X tiles.
      int pre = 0;
      auto load_b = [&](int st, int kb, int n_tile, int sub) {
        const uint32_t b_dst = smem_base + st * STAGE_BYTES + sub * (A_BYTES + B_BYTES) + A_BYTES;
        kb += sub;
        if (PAIR && hint) tma_load_2d_cg2_hint(b_dst, &tmap_x, lead_full(st), kb * BLK_K, n_tile * tokn + mrank * (tokn / 2), pol_x);
        else if (PAIR) tma_load_2d_cg2(b_dst, &tmap_x, lead_full(st), kb * BLK_K, n_tile * tokn + mrank * (tokn / 2));
        else if (hint) tma_load_2d_hint(b_dst, &tmap_x, full_bar(st), kb * BLK_K, n_tile * TOKN, pol_x);
        else tma_load_2d(b_dst, &tmap_x, full_bar(st), kb * BLK_K, n_tile * TOKN);
      };
      int w, kb0, kb1;
      trace_stamp(p, 12);
      {
        SegIter peek = segments();
        if (peek.next(w, kb0, kb1)) {            // the first segment's first stages (a later segment's are loaded in the loop)
          const int m_tile = m_tile_of(w);
          pre = p.tile_group ? 0 : min(STAGES * SUB, kb1 - kb0);      // which weights a tile needs is the previous kernel's output
          for (int i = 0; i * SUB < pre; ++i) {
            const int subs = min(SUB, kb1 - kb0 - i * SUB);
            expect(i, subs);
            for (int u = 0; u < subs; ++u) load_a(i, kb0 + i * SUB, m_tile, 0, u);
            if (i == 0) trace_stamp(p, 13);
          }
        }
      }
      trace_stamp(p, 2);
      pdl_wait();
      trace_stamp(p, 3);
      SegIter it = segments();
      bool first_seg = true;
      while (it.next(w, kb0, kb1)) {
        const int n_tile = w % p.n_tiles, m_tile = m_tile_of(w);
        if (no_rows(w)) continue;
        const int woff = p.tile_group ? p.tile_group[(n_tile * tokn) >> 8] * p.group_rows : 0;
        for (int kb = kb0; kb < kb1; kb += SUB) {
          const int subs = min(SUB, kb1 - kb);
          if (first_seg && kb - kb0 < pre) {
            for (int u = 0; u < subs; ++u) load_b(stage, kb, n_tile, u);
          } else {
            mbar_wait(empty_bar(stage), phase ^ 1);
            expect(stage, subs);
            for (int u = 0; u < subs; ++u) { load_a(stage, kb, m_tile, woff, u); load_b(stage, kb, n_tile, u); }
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        first_seg = false;
      }
      trace_stamp(p, 4);
    }
  } else if (warp == 1) {
    if ((!PAIR || mrank == 0) && elect_one()) {        // PAIR: the leader issues for both CTAs
      int stage = 0; uint32_t phase = 0;
      int acc = 0; uint32_t acc_phase = 0;
      SegIter it = segments();
      int w, kb0, kb1;
      if (p.trace) { mbar_wait(full_bar(0), 0); trace_stamp(p, 5); }      // (a wait does not consume the phase)
      // This one thread paces a decode-sized GEMM (every instruction between two k-blocks is serial latency), so the
      // loop carries the stage's descriptors along instead of rebuilding them.
      const uint64_t adesc0 = umma_desc_sw128(smem_base), bdesc0 = umma_desc_sw128(smem_base + A_BYTES);
      uint64_t adesc = adesc0, bdesc = bdesc0;
      while (it.next(w, kb0, kb1)) {
        if (no_rows(w)) continue;
        mbar_wait(tempty_bar(acc), acc_phase ^ 1);
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * TOKN;
        for (int kb = kb0; kb < kb1; kb += SUB) {
          mbar_wait(full_bar(stage), phase);
          tc_fence_after();
#pragma unroll
          for (int u = 0; u < SUB; ++u) {
            if (u > 0 && kb + u >= kb1) break;
#pragma unroll
            for (int k = 0; k < BLK_K / UMMA_K; ++k) {
              // +32 B per 16-element k step inside the 128 B swizzle row (start address field is >>4)
              const uint64_t off = (uint64_t)(u * ((A_BYTES + B_BYTES) >> 4) + k * 2);
              if (PAIR) tc_mma_bf16_cg2(d_tmem, adesc + off, bdesc + off, IDESC, (kb > kb0 || u + k > 0) ? 1u : 0u);
              else tc_mma_bf16(d_tmem, adesc + off, bdesc + off, IDESC, (kb > kb0 || u + k > 0) ? 1u : 0u);
            }
          }
          if (PAIR) tc_commit_cg2(empty_bar(stage), (uint16_t)(3u << leader)); // frees the stage in both CTAs
          else tc_commit(empty_bar(stage));     // frees the smem slot when these MMAs retire
          adesc += STAGE_BYTES >> 4; bdesc += STAGE_BYTES >> 4;
          if (++stage == STAGES) { stage = 0; phase ^= 1; adesc = adesc0; bdesc = bdesc0; }
        }
        if (PAIR) tc_commit_cg2(tfull_bar(acc), (uint16_t)(3u << leader));   // both CTAs' epilogues
        else tc_commit(tfull_bar(acc));         // accumulator complete
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      trace_stamp(p, 6);
    }
  } else if (warp >= 4) {
    const int q = warp - 4;                      // TMEM lane quarter == warp % 4
    const int et = threadIdx.x - 128;            // 0..127 == weight row within the tile
    int acc = 0; uint32_t acc_phase = 0;
    [[maybe_unused]] int hand = 0;               // GATED: which hand-off buffer is next
    SegIter it = segments();
    int w, kb0, kb1;
    while (it.next(w, kb0, kb1)) {
      const int n_tile = w % p.n_tiles, m_tile = m_tile_of(w);
      if (no_rows(w)) continue;
      const int t0 = n_tile * tokn;
      mbar_wait(tfull_bar(acc), acc_phase);
      tc_fence_after();
      if (et == 0) trace_stamp(p, 7);              // (of the CTA's last segment: later segments overwrite the stamp)
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * TOKN;
      if (WS && (kb0 != 0 || kb1 != KB)) {
        // ---- stream-K: this segment is only part of tile w's k range.  Its fp32 partial goes to the workspace
        // ([column][128 rows]: a warp stores 128 consecutive bytes per column); slot 0 of a CTA holds the partial that
        // STARTS its share, slot 1 the one that ends it.
        const int slot = ((int64_t)w * KB + kb0 == u_begin) ? 0 : 1;
        float* part = p.ws_part + ((int64_t)(blockIdx.x * 2 + slot) * TOKN) * BLK_M;
#pragma unroll 1
        for (int c = 0; c < TOKN; c += 16) {
          uint32_t r[16];
          tmem_ld16(taddr + c, r);
#pragma unroll
          for (int j = 0; j < 16; ++j) part[(c + j) * BLK_M + et] = __uint_as_float(r[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(acc));       // the accumulator is free: the next segment's MMAs may start
        __threadfence();                                   // the partial is visible device-wide before this CTA arrives
        asm volatile("bar.sync 1, 128;" ::: "memory");
        // which CTAs hold a part of tile w: the one containing its first unit ... the one containing its last unit
        const int64_t G = gridDim.x, x0 = (int64_t)w * KB, x1 = x0 + KB - 1;
        const int c_first = (int)(((x0 + 1) * G + U - 1) / U - 1), c_last = (int)(((x1 + 1) * G + U - 1) / U - 1);
        int* s_last = reinterpret_cast<int*>(tmem_slot + 1);
        if (et == 0) *s_last = (atomicAdd(p.ws_count + w, 1u) == (unsigned)(c_last - c_first)) ? 1 : 0;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (et == 0) trace_stamp(p, 8);
        if (*s_last) {
          // the LAST contributor to arrive reduces the tile: partials summed in k order (fixed), then the usual epilogue
          __threadfence();
          constexpr int QUADS = GATED ? 16 : 32;           // 4 consecutive weight rows per thread (GATED: + their up rows)
          constexpr int NGRP = 128 / QUADS;                // column groups
          constexpr int CPG = TOKN / NGRP;                 // columns per group
          constexpr int CH = CPG < 8 ? CPG : 8;            // columns held in registers at a time
          const int quad = et % QUADS, grp = et / QUADS;
          const int n0 = m_tile * ROWS_OUT + quad * 4;
          float bv4[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) bv4[k] = (p.bias && n0 + k < p.N) ? bf2f(p.bias[n0 + k]) : 0.f;
          const bool vec = (p.N & 3) == 0 && n0 + 3 < p.N;
#pragma unroll 1
          for (int cb = grp * CPG; cb < (grp + 1) * CPG; cb += CH) {
            float a[CH][4], u[GATED ? CH : 1][4];
#pragma unroll
            for (int ci = 0; ci < CH; ++ci) {
              a[ci][0] = a[ci][1] = a[ci][2] = a[ci][3] = 0.f;
              if (GATED) { u[ci][0] = u[ci][1] = u[ci][2] = u[ci][3] = 0.f; }
            }
            for (int cc = c_first; cc <= c_last; ++cc) {
              const int sl = (U * cc / G >= x0) ? 0 : 1;     // that CTA's share starts inside this tile: its slot 0
              const float* src = p.ws_part + ((int64_t)(cc * 2 + sl) * TOKN + cb) * BLK_M + quad * 4;
#pragma unroll
              for (int ci = 0; ci < CH; ++ci) {
                const float4 v = __ldcg(reinterpret_cast<const float4*>(src + ci * BLK_M));
                a[ci][0] += v.x; a[ci][1] += v.y; a[ci][2] += v.z; a[ci][3] += v.w;
                if (GATED) {
                  const float4 v2 = __ldcg(reinterpret_cast<const float4*>(src + ci * BLK_M + 64));
                  u[ci][0] += v2.x; u[ci][1] += v2.y; u[ci][2] += v2.z; u[ci][3] += v2.w;
                }
              }
            }
#pragma unroll
            for (int ci = 0; ci < CH; ++ci) {
              const int t = t0 + cb + ci;
              if (t < p.T) {
                float o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  if (GATED) o[k] = silu_gate_bf16(p, a[ci][k], u[ci][k], n0 + k);
                  else { o[k] = a[ci][k] + bv4[k]; o[k] = apply_act(o[k], p.act); }
                }
                bf16* dst = p.y + (int64_t)t * p.N + n0;
                if (vec) {
                  uint2 w2;
                  w2.x = pack_bf2(o[0], o[1]); w2.y = pack_bf2(o[2], o[3]);
                  *reinterpret_cast<uint2*>(dst) = w2;
                } else {
#pragma unroll
                  for (int k = 0; k < 4; ++k) if (n0 + k < p.N) dst[k] = f2bf(o[k]);
                }
              }
            }
          }
          if (et == 0) p.ws_count[w] = 0;                  // ready for the next launch
        }
      } else if (!XSPLIT) {
        // 32 tokens (columns) at a time: both 16-lane halves of this warp's rows come as MMA fragments, are finished and rounded
        // in registers, and stmatrix turns them into rows of 32 outputs per token in a staging tile of this warp's own, from where
        // a lane stores 16 bytes of an output row.  (One 2-byte store per output and a wait per 16 columns made the epilogue 10 us
        // of a single-wave launch: 1339 x 2048 x 2048 took 23 us, 10 of them in the main loop.)
        // GATED: gate rows live in warps q = 0, 1 and their up rows in q = 2, 3; each hands the other half of its tokens, rounded to
        // the element type as the product is, through shared memory.
        constexpr int G = TOKN >= 32 ? 4 : 2, CH = 8 * G;
        const uint32_t stage_buf = smem_addr(smem) + STAGES * STAGE_BYTES + 2048 + (GATED ? 8192 : 0) + q * 2048;
        uint32_t* swap = reinterpret_cast<uint32_t*>(xbuf);
        const int nq = m_tile * ROWS_OUT + (GATED ? (q & 1) : q) * 32;        // first output of this warp
        const bool vec = (p.N & 7) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0 && nq + 32 <= p.N;
        float bq[4];                                                          // bias of rows l / 4 + 8 i
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int nb = nq + 8 * i + (lane >> 2);
          bq[i] = p.bias && nb < p.N ? bf2f(p.bias[(GATED && q >= 2 ? p.N : 0) + nb]) : 0.f;
        }
        int c_begin = 0, c_end = tokn;
        const int share = SPLIT ? (tokn / 32 + S - 1) / S : 0;                // SPLIT: 32-token groups per pair of the cluster
        // [source][group of the owner's share][register quad][thread] of 16 bytes, over the pipeline stages
        auto xslot = [&](int src, int grp, int quad) { return smem_base + (uint32_t)((((src * share + grp) * 8 + quad) * 128 + et) * 16); };
        if constexpr (SPLIT) {
          cluster_arrive(); cluster_wait();                                   // no CTA of the cluster reads its stages any more
#pragma unroll 1
          for (int c = 0; c < tokn; c += CH) {
            const int grp = c / 32, owner = grp / share;
            if (owner == crank || t0 + c >= p.T) continue;
            uint32_t r[2][4 * G];
            tmem_ld_frag<G>(taddr + c, r[0]);
            tmem_ld_frag<G>(taddr + c + (16u << 16), r[1]);
            tmem_wait_ld(r[0], r[1]);
#pragma unroll
            for (int quad = 0; quad < 8; ++quad) {
              const uint32_t* v = &r[quad >> 2][(quad & 3) * 4];
              st_cluster_f4(mapa_u32(xslot(crank, grp - owner * share, quad), (uint32_t)(2 * owner + mrank)), __uint_as_float(v[0]), __uint_as_float(v[1]),
                            __uint_as_float(v[2]), __uint_as_float(v[3]));
            }
          }
          cluster_arrive(); cluster_wait();                                   // the owners have everything
          c_begin = crank * share * 32; c_end = min(tokn, c_begin + share * 32);
        }
#pragma unroll 1
        for (int c = c_begin; c < c_end; c += CH) {
          if (t0 + c >= p.T) break;                                           // the same for all epilogue warps
          uint32_t r[2][4 * G];
          tmem_ld_frag<G>(taddr + c, r[0]);
          tmem_ld_frag<G>(taddr + c + (16u << 16), r[1]);
          tmem_wait_ld(r[0], r[1]);
          if constexpr (SPLIT) {
            float sum[2][4 * G];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int i = 0; i < 4 * G; ++i) sum[h][i] = 0.f;
#pragma unroll 1
            for (int src = 0; src < S; ++src) {
#pragma unroll
              for (int quad = 0; quad < 8; ++quad) {
                float* d = &sum[quad >> 2][(quad & 3) * 4];
                const uint32_t* o = &r[quad >> 2][(quad & 3) * 4];
                const float4 f = src == crank ? make_float4(__uint_as_float(o[0]), __uint_as_float(o[1]), __uint_as_float(o[2]), __uint_as_float(o[3]))
                                              : lds_f4(xslot(src, (c - c_begin) / 32, quad));
                d[0] += f.x; d[1] += f.y; d[2] += f.z; d[3] += f.w;
              }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int i = 0; i < 4 * G; ++i) r[h][i] = __float_as_uint(sum[h][i]);
          }
          uint32_t o[G][4];                                                   // [8 tokens][8 rows]: two tokens of a row per register
          if (!GATED) {
            float v[2][4 * G];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int i = 0; i < 4 * G; ++i) v[h][i] = __uint_as_float(r[h][i]) + bq[2 * h + ((i >> 1) & 1)];
            if (p.act != 0) {
#pragma unroll
              for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 4 * G; ++i) v[h][i] = apply_act(v[h][i], p.act);
            }
#pragma unroll
            for (int k = 0; k < G; ++k)
#pragma unroll
              for (int i = 0; i < 4; ++i) o[k][i] = pack_bf2(v[i >> 1][4 * k + 2 * (i & 1)], v[i >> 1][4 * k + 2 * (i & 1) + 1]);
          } else {
            constexpr int HG = G / 2;
            const bool is_up = q >= 2;
            uint32_t mine[G][4];
#pragma unroll
            for (int k = 0; k < G; ++k)
#pragma unroll
              for (int i = 0; i < 4; ++i)
                mine[k][i] = pack_bf2(__uint_as_float(r[i >> 1][4 * k + 2 * (i & 1)]) + bq[i], __uint_as_float(r[i >> 1][4 * k + 2 * (i & 1) + 1]) + bq[i]);
            // [parity][pair][gate -> up, up -> gate][register][lane]
            uint32_t* hb = swap + (hand * 4 + (q & 1) * 2) * (8 * 32) + lane;
            hand ^= 1;                                                        // two buffers in turn, across tiles too
#pragma unroll
            for (int k = 0; k < HG; ++k)
#pragma unroll
              for (int i = 0; i < 4; ++i) hb[(is_up ? 256 : 0) + (k * 4 + i) * 32] = is_up ? mine[k][i] : mine[k + HG][i];
            asm volatile("bar.sync %0, 64;" ::"r"(2 + (q & 1)) : "memory");
#pragma unroll
            for (int k = 0; k < HG; ++k)
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint32_t other = hb[(is_up ? 0 : 256) + (k * 4 + i) * 32], own = is_up ? mine[k + HG][i] : mine[k][i];
                const uint32_t gv = is_up ? other : own, uv = is_up ? own : other;
                o[k][i] = pack_bf2(silu_gate_rounded(p, bf_lo(gv), bf_lo(uv)), silu_gate_rounded(p, bf_hi(gv), bf_hi(uv)));
              }
          }
          constexpr int OG = GATED ? G / 2 : G;                               // groups of 8 tokens that this warp stores
#pragma unroll
          for (int k = 0; k < OG; ++k) {
            const int tok = k * 8 + (lane & 7), piece = lane >> 3;
            stsm_trans(stage_buf + tok * 64 + ((piece ^ ((tok >> 1) & 3)) << 4), o[k][0], o[k][1], o[k][2], o[k][3]);
          }
          __syncwarp();
          const int tb = t0 + c + (GATED && q >= 2 ? CH / 2 : 0);
#pragma unroll
          for (int k = 0; k < OG; ++k) {
            const int tok = k * 8 + (lane >> 2), piece = lane & 3, t = tb + tok, n0 = nq + piece * 8;
            const float4 f = lds_f4(stage_buf + tok * 64 + ((piece ^ ((tok >> 1) & 3)) << 4));
            if (t < p.T) {
              bf16* dst = p.y + (int64_t)t * p.N + n0;
              if (vec) {
                *reinterpret_cast<float4*>(dst) = f;
              } else {
                const bf16* e = reinterpret_cast<const bf16*>(&f);
#pragma unroll
                for (int j = 0; j < 8; ++j) if (n0 + j < p.N) dst[j] = e[j];
              }
            }
          }
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { if (PAIR) mbar_arrive_cluster(mapa_u32(tempty_bar(acc), leader)); else mbar_arrive(tempty_bar(acc)); }
      } else {
        cluster_wait();                          // phase A done: peers' shared memory is live
        // Phase 1: my 128 x TOKN fp32 partial goes to the owners' exchange buffers, [src rank][local column][128 rows]:
        // one warp-wide store is 128 contiguous bytes of one remote column.
        const uint32_t xb = smem_addr(xbuf);
        {
          int owner = 0, lc = 0;
#pragma unroll 1
          for (int c = 0; c < TOKN; c += 16) {
            uint32_t r[16];
            tmem_ld16(taddr + c, r);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const uint32_t local = xb + (uint32_t)(((crank * cols_per + lc) * BLK_M + et) * 4);
              st_cluster_f32(mapa_u32(local, (uint32_t)owner), __uint_as_float(r[j]));
              if (++lc == cols_per) { lc = 0; ++owner; }
            }
          }
        }
        tc_fence_before();
        if (et == 0) trace_stamp(p, 8);
        cluster_arrive();                        // phase B: my partials are in the owners' buffers
        cluster_wait();
        if (et == 0) trace_stamp(p, 9);
        // Phase 2: my columns, summed over the ranks in rank order.  One item = 8 consecutive weight rows of one column:
        // 32 contiguous bytes per rank in shared memory, one 16-byte store of the output row.
        const int c_begin = crank * cols_per, c_end = min(TOKN, c_begin + cols_per);
        constexpr int RG = GATED ? 8 : 16;                       // 8-row groups per column
        const int n_items = (c_end - c_begin) * RG;
        const bool vec_ok = (p.N & 7) == 0;
        for (int item = et; item < n_items; item += 128) {
          const int lc = item / RG, rg = item % RG;
          const int t = t0 + c_begin + lc;
          if (t >= p.T) break;
          float a[8], u[GATED ? 8 : 1];
#pragma unroll
          for (int k = 0; k < 8; ++k) { a[k] = 0.f; if (GATED) u[k] = 0.f; }
          for (int s2 = 0; s2 < S; ++s2) {
            const uint32_t src = xb + (uint32_t)(((s2 * cols_per + lc) * BLK_M + rg * 8) * 4);
            const float4 v0 = lds_f4(src), v1 = lds_f4(src + 16);
            a[0] += v0.x; a[1] += v0.y; a[2] += v0.z; a[3] += v0.w;
            a[4] += v1.x; a[5] += v1.y; a[6] += v1.z; a[7] += v1.w;
            if (GATED) {
              const float4 w0 = lds_f4(src + 64 * 4), w1 = lds_f4(src + 64 * 4 + 16);
              u[0] += w0.x; u[1] += w0.y; u[2] += w0.z; u[3] += w0.w;
              u[4] += w1.x; u[5] += w1.y; u[6] += w1.z; u[7] += w1.w;
            }
          }
          const int n0 = m_tile * ROWS_OUT + rg * 8;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (GATED) {
              a[k] = silu_gate_bf16(p, a[k], u[k], n0 + k);
            } else {
              if (p.bias && n0 + k < p.N) a[k] += bf2f(p.bias[n0 + k]);
              a[k] = apply_act(a[k], p.act);
            }
          }
          bf16* dst = p.y + (int64_t)t * p.N + n0;
          if (vec_ok && n0 + 7 < p.N) {
            uint4 o;
            o.x = pack_bf2(a[0], a[1]); o.y = pack_bf2(a[2], a[3]); o.z = pack_bf2(a[4], a[5]); o.w = pack_bf2(a[6], a[7]);
            *reinterpret_cast<uint4*>(dst) = o;
          } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) if (n0 + k < p.N) dst[k] = f2bf(a[k]);
          }
        }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (et == 0) trace_stamp(p, 10);
  }
  if (SPLIT && warp < 4) {                       // non-epilogue warps take part in both cluster phases
    if (PAIR) cluster_arrive();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) trace_stamp(p, 11);
  if (PAIR) { cluster_arrive(); cluster_wait(); }   // the peer may still signal my barriers until it is done too
  if (warp == 2) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
  }
}

// ------------------------------------------------------------------------------ wide tiles for 33 to 64 tokens
// The operand roles swapped: the tokens are the M side (64 rows loaded; the MMA is 128 tall and its upper half reads whatever
// follows the token tile in shared memory - rows that are never read back), 256 weight rows are N of ONE MMA.  A token tile then
// goes with twice the weights, and a matrix of 43 to 74 tiles of 128 rows, which a split of K in two spreads over 86 to 148 CTAs,
// has 22 to 37 of these and a finer split.  D is [token][weight row] in TMEM: a thread owns a token and 256 consecutive outputs,
// which it stores 16 bytes at a time.  One tile per cluster, K split over its CTAs, the exchange buffer laid over the pipeline
// stages once every CTA of the cluster is past its main loop.
constexpr int WIDE_N = 256;                 // weight rows per tile
constexpr int WIDE_M = 64;                  // token rows per tile
constexpr uint32_t WIDE_A_BYTES = WIDE_M * BLK_K * 2, WIDE_B_BYTES = WIDE_N * BLK_K * 2;
constexpr uint32_t WIDE_STAGE = WIDE_A_BYTES + WIDE_B_BYTES;
constexpr int kWideStages = 5;
constexpr int kWideThreads = 384;           // warps 0-3 as in gemm_tc_kernel, two epilogue warpgroups

__global__ void __launch_bounds__(kWideThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const GemmParams p) {
  constexpr int STAGES = kWideStages;
  constexpr uint32_t TMEM_COLS = WIDE_N;
  constexpr uint32_t IDESC = (1u << 4) | KGE_IDESC_AB | ((uint32_t)(WIDE_N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  constexpr int UNIT = 16, N_UNITS = WIDE_N / UNIT;            // outputs per exchange unit

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * WIDE_STAGE);    // full[STAGES], empty[STAGES], tmem_full
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 2);
  const uint32_t smem_base = smem_addr(smem);
  const uint32_t bar_base = smem_addr(bars);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  const uint32_t tfull_bar = bar_base + 8u * (2 * STAGES);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) trace_stamp(p, 0);
  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
  }
  if (warp == 1 && lane == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(tfull_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) trace_stamp(p, 1);
  pdl_launch_dependents();
  if (warp != 0) pdl_wait();          // warp 0 (TMA producer) prefetches weights first, then waits

  const int S = (int)cluster_nctarank(), crank = (int)cluster_ctarank(), m_tile = (int)blockIdx.x / S;
  const int kb0 = crank * p.kb_per_split, kb1 = min(p.kb_total, kb0 + p.kb_per_split);
  const int n0 = m_tile * WIDE_N;                                               // first output column of the tile

  if (warp == 0) {
    if (elect_one()) {
      auto load_w = [&](int st, int kb) { tma_load_2d(smem_base + st * WIDE_STAGE + WIDE_A_BYTES, &tmap_w, full_bar(st), kb * BLK_K, n0); };
      trace_stamp(p, 12);
      const int pre = min(STAGES, kb1 - kb0);
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(full_bar(i), WIDE_STAGE);
        load_w(i, kb0 + i);
        if (i == 0) trace_stamp(p, 13);
      }
      trace_stamp(p, 2);
      pdl_wait();
      trace_stamp(p, 3);
      int stage = 0; uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (kb - kb0 >= pre) {
          mbar_wait(empty_bar(stage), phase ^ 1);
          mbar_expect_tx(full_bar(stage), WIDE_STAGE);
          load_w(stage, kb);
        }
        tma_load_2d(smem_base + stage * WIDE_STAGE, &tmap_x, full_bar(stage), kb * BLK_K, 0);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      trace_stamp(p, 4);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      if (p.trace) { mbar_wait(full_bar(0), 0); trace_stamp(p, 5); }
      int stage = 0; uint32_t phase = 0;
      const uint64_t adesc0 = umma_desc_sw128(smem_base), bdesc0 = umma_desc_sw128(smem_base + WIDE_A_BYTES);
      uint64_t adesc = adesc0, bdesc = bdesc0;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(full_bar(stage), phase);
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < BLK_K / UMMA_K; ++k)
          tc_mma_bf16(tmem_base, adesc + (uint64_t)(k * 2), bdesc + (uint64_t)(k * 2), IDESC, (kb > kb0 || k > 0) ? 1u : 0u);
        tc_commit(empty_bar(stage));
        adesc += WIDE_STAGE >> 4; bdesc += WIDE_STAGE >> 4;
        if (++stage == STAGES) { stage = 0; phase ^= 1; adesc = adesc0; bdesc = bdesc0; }
      }
      tc_commit(tfull_bar);
      trace_stamp(p, 6);
    }
  }
  else if (warp >= 4) {
    // Two epilogue warpgroups (warps 4-7, 8-11): a warp reads the TMEM lane quarter warp % 4, the tokens live in lanes
    // 0-63, so warps 4, 5 take the first half of the tile's units for their tokens and warps 8, 9 the second half; all
    // eight warps share the reduction of the split variant.
    const int et = threadIdx.x - 128, q = warp & 3, eg = (warp - 4) >> 2;
    const int tok = q * 32 + lane;                          // my token (TMEM lane) if q < 2
    const int u_half = (N_UNITS + 1) / 2;
    const int u_lo = eg * u_half, u_hi = eg ? N_UNITS : u_half;
    mbar_wait(tfull_bar, 0);
    tc_fence_after();
    if (et == 0) trace_stamp(p, 7);
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
    const bool vec_ok = (p.N & 7) == 0;
    // the 16 outputs of unit u from raw accumulators: bias, activation
    auto finish = [&](int u, const float (&a)[16], float (&o)[16]) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int n = n0 + u * UNIT + j;
        o[j] = apply_act(a[j] + ((p.bias && n < p.N) ? bf2f(p.bias[n]) : 0.f), p.act);
      }
    };
    auto store16 = [&](int t, int u, const float (&o)[16]) {
      if (t >= p.T) return;
      const int n = n0 + u * UNIT;
      bf16* dst = p.y + (int64_t)t * p.N + n;
      if (vec_ok && n + 15 < p.N) {
        uint4 w0, w1;
        w0.x = pack_bf2(o[0], o[1]); w0.y = pack_bf2(o[2], o[3]); w0.z = pack_bf2(o[4], o[5]); w0.w = pack_bf2(o[6], o[7]);
        w1.x = pack_bf2(o[8], o[9]); w1.y = pack_bf2(o[10], o[11]); w1.z = pack_bf2(o[12], o[13]); w1.w = pack_bf2(o[14], o[15]);
        reinterpret_cast<uint4*>(dst)[0] = w0;
        reinterpret_cast<uint4*>(dst)[1] = w1;
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) if (n + j < p.N) dst[j] = f2bf(o[j]);
      }
    };
    const int units_per = (N_UNITS + S - 1) / S;
    constexpr int NJ = UNIT / 4;                            // 16-byte pieces of a unit
    // exchange buffer of a CTA: [source rank][local unit][piece][token][4 fp32] - a warp stores (and later loads) 512
    // contiguous bytes
    const uint32_t xb = smem_base;                          // over the pipeline stages: dead once phase A completes
    cluster_arrive();                                       // phase A: my MMAs have read their last stage
    cluster_wait();
    if (q < 2) {
#pragma unroll 1
      for (int u = u_lo; u < u_hi; ++u) {
        uint32_t r[16];
        tmem_ld16(taddr + u * UNIT, r);
        const int owner = u / units_per, lu = u - owner * units_per;
        const uint32_t dst = mapa_u32(xb + (uint32_t)(((((crank * units_per + lu) * NJ) * WIDE_M) + tok) * 16), (uint32_t)owner);
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          st_cluster_f4(dst + j * (WIDE_M * 16), __uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
      }
    }
    tc_fence_before();
    if (et == 0) trace_stamp(p, 8);
    cluster_arrive();                                       // phase B: my partials are in the owners' buffers
    cluster_wait();
    if (et == 0) trace_stamp(p, 9);
    // my units, summed over the ranks in rank order; one item = one token's 16 outputs of one unit
    const int u_begin = crank * units_per;
    const int my_units = min(N_UNITS, u_begin + units_per) - u_begin;
    for (int item = et; item < my_units * WIDE_M; item += 256) {
      const int t = item & (WIDE_M - 1), lu = item / WIDE_M;
      float a[16], o[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) a[j] = 0.f;
      for (int s2 = 0; s2 < S; ++s2) {
        const uint32_t src = xb + (uint32_t)(((((s2 * units_per + lu) * NJ) * WIDE_M) + t) * 16);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float4 v = lds_f4(src + j * (WIDE_M * 16));
          a[4 * j] += v.x; a[4 * j + 1] += v.y; a[4 * j + 2] += v.z; a[4 * j + 3] += v.w;
        }
      }
      finish(u_begin + lu, a, o);
      store16(t, u_begin + lu, o);
    }
    if (et == 0) trace_stamp(p, 10);
  }
  if (warp < 4) {                       // non-epilogue warps take part in both cluster phases
    cluster_arrive();
    cluster_wait();
    cluster_arrive();
    cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) trace_stamp(p, 11);
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
  }
}

// ------------------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* ptr = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(ptr);
  return fn;
}

// 2-D row-major bf16 [rows, cols] with a {64 x box_rows} box and 128B swizzle.
static int encode_tmap(CUtensorMap* m, const void* ptr, int64_t rows, int64_t cols, int box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  KGE_REQUIRE(enc, "cuTensorMapEncodeTiled unavailable (no CUDA driver?)");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {(cuuint32_t)BLK_K, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
#ifdef KGE_HALF
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
#else
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
#endif
  CUresult r = enc(m, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  KGE_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d) rows=%lld cols=%lld", (int)r, (long long)rows, (long long)cols);
  return 0;
}

// A tensor map is a pure function of (address, shape, box): the engine's weights and activation buffers keep their
// addresses, so each map is encoded once and looked up afterwards (two host-side driver calls per GEMM launch otherwise,
// which is what an un-graphed step pays on every one of its ~200 GEMMs).
struct TmapKey {
  const void* p; int64_t rows, cols; int box;
  bool operator==(const TmapKey& o) const { return p == o.p && rows == o.rows && cols == o.cols && box == o.box; }
};
struct TmapKeyHash {
  size_t operator()(const TmapKey& k) const {
    uint64_t h = (uint64_t)(uintptr_t)k.p * 0x9E3779B97F4A7C15ull;
    h ^= ((uint64_t)k.rows * 0xBF58476D1CE4E5B9ull) ^ ((uint64_t)k.cols << 20) ^ (uint64_t)k.box;
    return (size_t)(h ^ (h >> 29));
  }
};
// Tensor maps by what they are made of, for all threads.  Callers that cycle through fresh buffers (tests) stay bounded.
template <class Key, class Hash, class Encode>
static int cached_tmap(CUtensorMap* m, const Key& key, Encode&& encode) {
  static std::mutex mu;
  static std::unordered_map<Key, CUtensorMap, Hash> cache;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(key);
  if (it != cache.end()) { *m = it->second; return 0; }
  if (int rc = encode(m)) return rc;
  if (cache.size() >= 16384) cache.clear();
  cache.emplace(key, *m);
  return 0;
}
int make_tmap(CUtensorMap* m, const void* ptr, int64_t rows, int64_t cols, int box_rows) {
  return cached_tmap<TmapKey, TmapKeyHash>(m, TmapKey{ptr, rows, cols, box_rows}, [&](CUtensorMap* t) { return encode_tmap(t, ptr, rows, cols, box_rows); });
}

// Queries of a packed projection, [tokens][heads][hd] with tokens `stride` numbers apart: boxes of 64 columns x box_heads x
// box_tokens, 128B swizzle.  The number of tokens is not known to the callers: a box must lie within the rows they may read.
static int encode_tmap_q(CUtensorMap* m, const void* ptr, int64_t stride, int hd, int heads, int box_heads, int box_tokens) {
  EncodeTiledFn enc = get_encode_fn();
  KGE_REQUIRE(enc, "cuTensorMapEncodeTiled unavailable (no CUDA driver?)");
  cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)heads, (cuuint64_t)1 << 30};
  cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)stride * 2};
  cuuint32_t box[3] = {64, (cuuint32_t)box_heads, (cuuint32_t)box_tokens};
  cuuint32_t estr[3] = {1, 1, 1};
#ifdef KGE_HALF
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
#else
  const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
#endif
  CUresult r = enc(m, dt, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  KGE_REQUIRE(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed (%d) stride=%lld heads=%d", (int)r, (long long)stride, heads);
  return 0;
}

struct TmapQKey {
  const void* p; int64_t stride; int hd, heads, box_heads, box_tokens;
  bool operator==(const TmapQKey& o) const { return p == o.p && stride == o.stride && hd == o.hd && heads == o.heads && box_heads == o.box_heads && box_tokens == o.box_tokens; }
};
struct TmapQKeyHash {
  size_t operator()(const TmapQKey& k) const {
    uint64_t h = (uint64_t)(uintptr_t)k.p * 0x9E3779B97F4A7C15ull;
    h ^= ((uint64_t)k.stride * 0xBF58476D1CE4E5B9ull) ^ ((uint64_t)k.heads << 40) ^ ((uint64_t)k.hd << 24) ^ ((uint64_t)k.box_heads << 8) ^ (uint64_t)k.box_tokens;
    return (size_t)(h ^ (h >> 29));
  }
};
int make_tmap_q(CUtensorMap* m, const void* ptr, int64_t stride, int hd, int heads, int box_heads, int box_tokens) {
  return cached_tmap<TmapQKey, TmapQKeyHash>(m, TmapQKey{ptr, stride, hd, heads, box_heads, box_tokens},
                                             [&](CUtensorMap* t) { return encode_tmap_q(t, ptr, stride, hd, heads, box_heads, box_tokens); });
}

constexpr int kGemmSmemBudget = 224 * 1024;

template <int TOKN, bool SPLIT, bool GATED, bool PAIR = false, bool WS = false>
static int launch_gemm(const CUtensorMap& tw, const CUtensorMap& tx, const GemmParams& p, cudaStream_t st) {
  constexpr int stage_bytes = (BLK_M * BLK_K * 2 + (PAIR ? 128 : TOKN) * BLK_K * 2) * (PAIR ? kPairSub : 1);
  // barriers, then the cluster exchange buffer (SPLIT), or the gate / up hand-off (GATED) and the epilogue's staging tiles
  constexpr int extra = 2048 + (SPLIT && !PAIR ? xbuf_bytes(TOKN) : (GATED ? 8192 : 0) + 8192);
  constexpr int budget = kGemmSmemBudget - 1024 - extra;
  constexpr int STAGES = (budget / stage_bytes) > 8 ? 8 : (budget / stage_bytes);
  static_assert(STAGES >= 3, "pipeline too shallow");
  constexpr int smem = STAGES * stage_bytes + 1024 /*align*/ + extra;
  auto kern = gemm_tc_kernel<TOKN, STAGES, SPLIT, GATED, PAIR, WS>;
  KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  prefer_max_shared(kern);
  const int tiles = p.m_tiles * p.n_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_for_this_launch() ? 1 : 0;
  cfg.attrs = attr; cfg.numAttrs = 1;
  if (WS) {
    cfg.gridDim = dim3(p.splits);                // stream-K: `splits` CTAs (one per SM), each a contiguous share of all k-blocks
  } else if (SPLIT) {
    const int ctas = PAIR ? 2 * p.splits : p.splits;
    cfg.gridDim = dim3((PAIR ? (p.m_tiles + 1) / 2 * p.n_tiles : tiles) * ctas);
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ctas; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  } else if (PAIR) {
    const int pairs = ((p.m_tiles + 1) / 2) * p.n_tiles;
    cfg.gridDim = dim3(2 * (pairs < 74 ? pairs : 74));
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  } else {
    constexpr int slots = 148;
    int grid = tiles < slots ? tiles : slots;
    if (tunable(TUN_GEMM_EVEN_GRID) && tiles > 148) {
      // persistent round-robin: 224 tiles on 148 CTAs leaves 72 CTAs idle for the second half; 112 CTAs with two
      // tiles each keep every CTA streaming to the end (a weight-streaming GEMM needs bytes in flight, not SMs)
      const int rounds = (tiles + 147) / 148;
      grid = (tiles + rounds - 1) / rounds;
    }
    cfg.gridDim = dim3(grid);
  }
  KGE_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tw, tx, p));
  return 0;
}

template <int TOKN>
static int query_max_clusters(int S) {
  constexpr int stage_bytes = BLK_M * BLK_K * 2 + TOKN * BLK_K * 2;
  constexpr int extra = 2048 + xbuf_bytes(TOKN);
  constexpr int budget = kGemmSmemBudget - 1024 - extra;
  constexpr int STAGES = (budget / stage_bytes) > 8 ? 8 : (budget / stage_bytes);
  constexpr int smem = STAGES * stage_bytes + 1024 + extra;
  auto kern = gemm_tc_kernel<TOKN, STAGES, true, false>;   // the gated variant has the same footprint
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S * 64); cfg.blockDim = dim3(kGemmThreads); cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  return n;
}

// How many clusters of size S of the split kernel can be co-resident (GPC packing decides: 148 SMs
// hold e.g. 34 clusters of 4 but fewer than 148/3 clusters of 3).  Cached per (token tile, S).
static int max_clusters(int tokn, int S) {
  static int cache[4][9];
  static bool have[4][9];
  const int ti = tokn == 16 ? 0 : tokn == 32 ? 1 : tokn == 64 ? 2 : 3;
  if (!have[ti][S]) {
    cache[ti][S] = ti == 0 ? query_max_clusters<16>(S) : ti == 1 ? query_max_clusters<32>(S)
                 : ti == 2 ? query_max_clusters<64>(S) : query_max_clusters<128>(S);
    have[ti][S] = true;
  }
  return cache[ti][S];
}

struct GemmPlan { int tokn, m_tiles, n_tiles, splits, kb_total, kb_per_split; bool ws; bool pair = false; };

constexpr int64_t kWsCounterBytes = 1024;        // per-tile arrival counters at the head of the workspace (<= 256 tiles)

// ws_ok: the caller can provide a workspace, so split-K may go through it (two CTAs per SM) instead of a cluster
static GemmPlan plan_gemm(int T, int N, int K, int rows_out = BLK_M, bool ws_ok = false) {
  GemmPlan g;
  g.ws = false;
  g.tokn = T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : T <= 128 ? 128 : 256;
  g.m_tiles = (N + rows_out - 1) / rows_out;
  g.n_tiles = (T + g.tokn - 1) / g.tokn;
  g.kb_total = (K + BLK_K - 1) / BLK_K;
  const int tiles = g.m_tiles * g.n_tiles;
  int splits = 1;
  const int slots = 148;                       // CTAs that can be resident at once
  if (ws_ok && g.tokn <= 128 && tiles <= (int)(kWsCounterBytes / 4) && tiles % 148 != 0 && tunable(TUN_GEMM_WS)) {
    // stream-K: one CTA per SM, every CTA the same number of k-blocks (at least 4, i.e. 256 of K)
    const int64_t units = (int64_t)tiles * g.kb_total;
    int ctas = units / 4 < 148 ? (int)(units / 4) : 148;
    if (ctas >= 2) { g.ws = true; splits = ctas; }
  }
  if (!g.ws && tiles <= slots / 2 && g.tokn <= 128) {
    int smax = slots / tiles;                   // never more CTAs than resident slots
    const int max_by_k = g.kb_total / 4 > 0 ? g.kb_total / 4 : 1;   // >= 4 k-blocks (256 of K) per split
    if (smax > max_by_k) smax = max_by_k;
    if (smax > 8) smax = 8;                     // portable cluster size
    for (int s = smax; s >= 2; --s)             // largest S whose clusters all fit in ONE wave
      if (tiles <= max_clusters(g.tokn, s)) { splits = s; break; }
  }
  if (g.ws) { g.kb_per_split = g.kb_total; g.splits = splits; return g; }      // `splits` carries the grid size
  g.kb_per_split = (g.kb_total + splits - 1) / splits;
  g.splits = (g.kb_total + g.kb_per_split - 1) / g.kb_per_split;   // drop empty splits
  return g;
}

// ---- wide tiles: one tile of 256 weight rows per cluster
constexpr int kWideSmem = kWideStages * (int)WIDE_STAGE + 1024 /*align*/ + 2048 /*barriers*/;

static int launch_wide(const CUtensorMap& tw, const CUtensorMap& tx, const GemmParams& p, cudaStream_t st) {
  KGE_CUDA_OK(cudaFuncSetAttribute(gemm_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem));
  prefer_max_shared(gemm_wide_kernel);
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kWideThreads);
  cfg.dynamicSmemBytes = kWideSmem;
  cfg.stream = st;
  cfg.gridDim = dim3(p.m_tiles * p.splits);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_for_this_launch() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = p.splits; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  KGE_CUDA_OK(cudaLaunchKernelEx(&cfg, gemm_wide_kernel, tw, tx, p));
  return 0;
}

static int max_clusters_wide(int S) {
  static int cache[9];
  static bool have[9];
  if (!have[S]) {
    auto kern = gemm_wide_kernel;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(S * 64); cfg.blockDim = dim3(kWideThreads); cfg.dynamicSmemBytes = kWideSmem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr; cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
    }
    cache[S] = n; have[S] = true;
  }
  return cache[S];
}

// Whether a projection takes the wide tiles, and the K split: the largest whose clusters fit one round.  Only 33 to 64 tokens where
// the 128-row plan splits K in two: us with wide and 128-row tiles, 64 tokens, 8192 x 8192 26.1 / 27.3, 7168 x 2048 9.9 / 10.2,
// 6144 x 4096 13.6 / 13.8; up to 32 tokens a token tile is too small to matter (6144 x 4096 13.5 / 12.4), a split in three is finer
// than what clusters of 256 rows leave (5120 x 5120 14.1 / 13.0), and more than 74 tiles need no split (16384 x 2048 15.4 / 13.4,
// 28672 x 4096 42.0 / 40.2, gated 45.1 / 41.0, gated 16384 x 2048 16.8 / 13.9).
static bool plan_wide(int T, int n_out, int K, GemmPlan& g) {
  if (!tunable(TUN_GEMM_WIDE) || T > WIDE_M || T <= WIDE_M / 2 || plan_gemm(T, n_out, K).splits != 2) return false;
  g.kb_total = (K + BLK_K - 1) / BLK_K;
  g.m_tiles = (n_out + WIDE_N - 1) / WIDE_N;
  int sp = 148 / g.m_tiles;
  if (sp > g.kb_total / 4) sp = g.kb_total / 4;        // >= 4 k-blocks (256 of K) per split
  if (sp > 8) sp = 8;
  while (sp > 1 && g.m_tiles > max_clusters_wide(sp)) --sp;
  if (sp < 2) return false;
  g.ws = false;
  g.tokn = WIDE_M; g.n_tiles = 1;
  g.kb_per_split = (g.kb_total + sp - 1) / sp;
  g.splits = (g.kb_total + g.kb_per_split - 1) / g.kb_per_split;
  return true;
}

#include "gemm_rows.cuh"

// How many clusters of `size` CTAs of the pair kernel can be co-resident.
static int max_clusters_pair(int size) {
  static std::atomic<int> cache[9];
  int n = cache[size].load(std::memory_order_relaxed);
  if (n == 0) {
    constexpr int stage_bytes = 2 * BLK_M * BLK_K * 2 * kPairSub, extra = 2048 + 8192, STAGES = (kGemmSmemBudget - 1024 - extra) / stage_bytes;
    constexpr int smem = STAGES * stage_bytes + 1024 + extra;
    auto kern = gemm_tc_kernel<256, STAGES, true, false, true>;
    int got = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(size * 64); cfg.blockDim = dim3(kGemmThreads); cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = size; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr; cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&got, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); got = 0; }
    }
    n = got + 1;
    cache[size].store(n, std::memory_order_relaxed);
  }
  return n - 1;
}

// More than 64 tokens run as CTA pairs (cta_group::2, 256 weight rows x up to 256 tokens).  The width of the token tile and the
// split of K are those with the least estimated time, fitted to measurements: a k-block takes 0.235 us and 0.055 more for a full
// 256 tokens (data and MMAs; narrow tiles are hardly faster, so what a narrow tile saves is an empty last round), a launch 3.9 us
// and up to 3.3 for the epilogue of the last tile, an exchange 1.2 per further share and up to 2.  us with tiles of 256 and K
// whole, and now: 200 x 4096 x 4096 23.5 / 14.9, 256 x 4096 x 14336 71.7 / 37.7, 700 x 2048 x 8192 49 / 24.5, 1339 x 2048 x 2048
// 15.8 / 13.7, 2312 x 2048 x 8192 82.5 / 70.5, 333 x 6144 x 4096 24.7 / 22.1.
// Up to 128 tokens the single-CTA kernel keeps what it splits into four shares of K or more (128 x 2048 x 8192: 14.3 us, 16.1 here).
// fixed: the token tile has to be 256 wide and K whole (grouped rows).
static bool plan_pairs(int T, int n_out, int K, int rows_out, bool fixed, GemmPlan& g) {
  if (T <= 128 && g.splits >= 4) return false;
  const int m_tiles = (n_out + rows_out - 1) / rows_out, kb_total = (K + BLK_K - 1) / BLK_K;
  if (T <= WIDE_M || m_tiles < 2) return false;
  const int pairs = (m_tiles + 1) / 2;
  double best = 1e30;
  for (int S = 1; S <= (fixed ? 1 : 4); ++S) {
    if (S > 1 && kb_total / S < 4) break;
    const int kb = (kb_total + S - 1) / S;
    for (int tokn = 256; tokn >= (fixed ? 256 : 32); tokn -= 32) {
      const int64_t tiles = (int64_t)pairs * ((T + tokn - 1) / tokn);
      if (S > 1 && tiles > max_clusters_pair(2 * S)) break;              // narrower tiles are more tiles
      const int64_t rounds = S > 1 ? 1 : (tiles + 73) / 74;
      const double us = rounds * (kb * (0.235 + 0.055 * tokn / 256) + 0.3) + 3.9 + 3.3 * tokn / 256 + (S > 1 ? 1.2 * (S - 1) + 2.0 * tokn / 256 : 0.0);
      if (us < best) {
        best = us;
        g.tokn = tokn; g.splits = S;
      }
    }
  }
  g.ws = false; g.pair = true;
  g.m_tiles = m_tiles; g.n_tiles = (T + g.tokn - 1) / g.tokn;
  g.kb_total = kb_total; g.kb_per_split = (kb_total + g.splits - 1) / g.splits;
  g.splits = (kb_total + g.kb_per_split - 1) / g.kb_per_split;           // drop empty splits
  return true;
}

template <bool GATED>
static int dispatch_gemm(const GemmPlan& g, const CUtensorMap& tw, const CUtensorMap& tx, const GemmParams& p, cudaStream_t st) {
  if (g.pair) return g.splits > 1 ? launch_gemm<256, true, GATED, true>(tw, tx, p, st) : launch_gemm<256, false, GATED, true>(tw, tx, p, st);
  if (g.ws) {
    switch (g.tokn) {
      case 16: return launch_gemm<16, false, GATED, false, true>(tw, tx, p, st);
      case 32: return launch_gemm<32, false, GATED, false, true>(tw, tx, p, st);
      case 64: return launch_gemm<64, false, GATED, false, true>(tw, tx, p, st);
      default: return launch_gemm<128, false, GATED, false, true>(tw, tx, p, st);
    }
  }
  if (g.splits > 1) {
    switch (g.tokn) {
      case 16: return launch_gemm<16, true, GATED>(tw, tx, p, st);
      case 32: return launch_gemm<32, true, GATED>(tw, tx, p, st);
      case 64: return launch_gemm<64, true, GATED>(tw, tx, p, st);
      default: return launch_gemm<128, true, GATED>(tw, tx, p, st);
    }
  }
  switch (g.tokn) {
    case 16: return launch_gemm<16, false, GATED>(tw, tx, p, st);
    case 32: return launch_gemm<32, false, GATED>(tw, tx, p, st);
    case 64: return launch_gemm<64, false, GATED>(tw, tx, p, st);
    case 128: return launch_gemm<128, false, GATED>(tw, tx, p, st);
    default:
      return launch_gemm<256, false, GATED>(tw, tx, p, st);
  }
}

}  // namespace KGE_ELT_NS
}  // namespace kge

using namespace kge;

#ifndef KGE_HALF
unsigned long long* g_gemm_trace = nullptr;
// Measurement hook of tools/gemm_trace.py: device buffer of 16 timestamps per CTA of the following GEMM launches
// (both element types), or null to stop.  No counterpart in the reference.
extern "C" void kge_gemm_set_trace(void* device_buffer) { g_gemm_trace = (unsigned long long*)device_buffer; }
#else
extern unsigned long long* g_gemm_trace;
#endif

static int64_t ws_bytes_of(const GemmPlan& g) {        // counters + two partial tiles per CTA
  return g.ws ? kWsCounterBytes + (int64_t)g.splits * 2 * g.tokn * BLK_M * 4 : 0;
}

#ifndef KGE_HALF      // the same for both element types: exported once
extern "C" int64_t kge_gemm_workspace_bytes(int T, int N, int K) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  // enough for the plain projection and for the fused SiLU-gate one with f = N (64 output rows per tile); 0: this shape
  // does not go through a workspace
  const int64_t a = ws_bytes_of(plan_gemm(T, N, K, BLK_M, true)), b = ws_bytes_of(plan_gemm(T, N, K, 64, true));
  return a > b ? a : b;
}

#endif

#ifdef KGE_HALF
#define KGE_GEMM_NAME kge_gemm_f16
#define KGE_GEMM_GATE_NAME kge_gemm_silu_gate_f16
#define KGE_GEMM_GATE_WS_NAME kge_gemm_silu_gate_ws_f16
#define KGE_GEMM_GLU_NAME kge_gemm_clamped_glu_f16
#else
#define KGE_GEMM_NAME kge_gemm_bf16
#define KGE_GEMM_GATE_NAME kge_gemm_silu_gate_bf16
#define KGE_GEMM_GATE_WS_NAME kge_gemm_silu_gate_ws_bf16
#define KGE_GEMM_GLU_NAME kge_gemm_clamped_glu_bf16
#endif
// Up to 8 rows of up to 1024, and outputs for no more CTAs than are resident at once: norm and projection in two launches and in one,
// us, 768 x 2304 at 1 and 8 tokens 4.0 / 3.2 and 4.7 / 3.7, 768 x 3072 3.6 / 3.3 and 4.2 / 3.9, 1024 x 4096 3.7 / 3.5 and 4.25 / 4.25.
// Longer rows and more CTAs pay for a norm in each CTA (2048 x 3072 4.9 / 6.4, 2048 x 6144 8.7 / 15.0).
#ifndef KGE_HALF
extern "C" bool kge_norm_gemm_ok(int T, int N, int K) {
  return T > 0 && T <= 8 && K % 8 == 0 && K <= 32 * 8 * kNormVecs && N <= 2 * 148 * 16 && use_rows(T, N, K);
}
#endif
extern "C" int KGE_API(kge_norm_gemm)(void* y, const RowsNorm& nm, const void* w, const void* bias, int T, int N, int K, int act, const RowsKv& kv, void* stream) {
  KGE_REQUIRE(kge_norm_gemm_ok(T, N, K) && (!nm.add || (nm.res_out && nm.res_out != nm.res)), "kge_norm_gemm: sizes");
  GemmParams p;
  p.y = (bf16*)y; p.bias = (const bf16*)bias; p.T = T; p.N = N; p.K = K; p.act = act;
  return N < 16 * 148 ? launch_norm_rows<1, 4>((const bf16*)w, p, nm, kv, (cudaStream_t)stream) : launch_norm_rows<2, 3>((const bf16*)w, p, nm, kv, (cudaStream_t)stream);
}

extern "C" int KGE_GEMM_NAME(void* y, const void* x, const void* w, const void* bias, int T, int N, int K,
                             int act, void* workspace, int64_t workspace_bytes, void* stream) {
  KGE_REQUIRE(y && x && w, "kge_gemm_bf16: null pointer");
  KGE_REQUIRE(T >= 0 && N > 0 && K > 0 && K % 8 == 0, "kge_gemm_bf16: K=%d must be a positive multiple of 8", K);
  KGE_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0, "kge_gemm_bf16: x and w must be 16-byte aligned");
  KGE_REQUIRE(act == 0 || act == 1 || act == 3 || act == 4, "kge_gemm_bf16: act=%d unsupported (0 none, 1 relu, 3 gelu, 4 squared relu)", act);
  if (T == 0) return 0;
  bool use_ws = workspace && tunable(TUN_GEMM_WS);          // stream-K through the caller's scratch, if it is large enough
  if (use_ws) {
    const GemmPlan gq = plan_gemm(T, N, K, BLK_M, true);
    use_ws = gq.ws && workspace_bytes >= ws_bytes_of(gq) && ((uintptr_t)workspace & 15) == 0;
  }
  if (!use_ws) {
    if (use_rows(T, N, K)) {
      GemmParams p;
      p.y = (bf16*)y; p.bias = (const bf16*)bias; p.T = T; p.N = N; p.K = K; p.act = act;
      return launch_rows<false>((const bf16*)x, (const bf16*)w, p, (cudaStream_t)stream);
    }
    GemmPlan gw;
    if (plan_wide(T, N, K, gw)) {
      GemmParams p;
      p.y = (bf16*)y; p.bias = (const bf16*)bias; p.T = T; p.N = N; p.K = K; p.act = act;
      p.l2_hints = 0; p.trace = g_gemm_trace; p.ws_count = nullptr; p.ws_part = nullptr;
      p.m_tiles = gw.m_tiles; p.n_tiles = 1; p.splits = gw.splits; p.kb_total = gw.kb_total; p.kb_per_split = gw.kb_per_split;
      CUtensorMap tw, tx;
      if (int rc = make_tmap(&tw, w, N, K, WIDE_N)) return rc;
      if (int rc = make_tmap(&tx, x, T, K, WIDE_M)) return rc;
      return launch_wide(tw, tx, p, (cudaStream_t)stream);
    }
  }
  GemmPlan g = plan_gemm(T, N, K, BLK_M, workspace != nullptr);
  if (g.ws && (workspace_bytes < ws_bytes_of(g) || ((uintptr_t)workspace & 15) != 0))
    g = plan_gemm(T, N, K);                        // scratch too small for this shape: split K inside a cluster instead
  if (!g.ws) (void)plan_pairs(T, N, K, BLK_M, false, g);
  GemmParams p;
  p.y = (bf16*)y; p.bias = (const bf16*)bias; p.T = T; p.N = N; p.K = K; p.act = act;
  p.l2_hints = tunable(TUN_GEMM_L2_HINTS);
  p.trace = g_gemm_trace;
  p.ws_count = g.ws ? (unsigned int*)workspace : nullptr;
  p.ws_part = g.ws ? (float*)((uint8_t*)workspace + kWsCounterBytes) : nullptr;
  p.m_tiles = g.m_tiles; p.n_tiles = g.n_tiles; p.splits = g.splits;
  p.kb_total = g.kb_total; p.kb_per_split = g.kb_per_split; p.tokn = g.tokn;
  CUtensorMap tw, tx;
  if (int rc = make_tmap(&tw, w, N, K, BLK_M)) return rc;
  if (int rc = make_tmap(&tx, x, T, K, g.pair ? g.tokn / 2 : g.tokn)) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  return dispatch_gemm<false>(g, tw, tx, p, st);
}

static int gemm_gated(void* y, const void* x, const void* w_gate_up, int T, int f, int K, int glu, float glu_alpha, float glu_limit, void* workspace,
                      int64_t workspace_bytes, void* stream, const void* bias_gate_up = nullptr) {
  KGE_REQUIRE(y && x && w_gate_up, "kge_gemm_silu_gate_bf16: null pointer");
  KGE_REQUIRE(T >= 0 && f > 0 && K > 0 && K % 8 == 0, "kge_gemm_silu_gate_bf16: K=%d must be a positive multiple of 8", K);
  KGE_REQUIRE(f % 64 == 0, "kge_gemm_silu_gate_bf16: f=%d must be a multiple of 64", f);
  KGE_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)w_gate_up & 15) == 0, "kge_gemm_silu_gate_bf16: x and w must be 16-byte aligned");
  if (T == 0) return 0;
  bool use_ws = workspace && tunable(TUN_GEMM_WS);
  if (use_ws) {
    const GemmPlan gq = plan_gemm(T, f, K, 64, true);
    use_ws = gq.ws && workspace_bytes >= ws_bytes_of(gq) && ((uintptr_t)workspace & 15) == 0;
  }
  if (!use_ws) {
    if (use_rows(T, 2 * f, K)) {
      GemmParams p;
      p.y = (bf16*)y; p.bias = (const bf16*)bias_gate_up; p.T = T; p.N = f; p.K = K; p.act = 2; p.glu = glu; p.glu_alpha = glu_alpha; p.glu_limit = glu_limit;
      return launch_rows<true>((const bf16*)x, (const bf16*)w_gate_up, p, (cudaStream_t)stream);
    }
  }
  GemmPlan g = plan_gemm(T, f, K, 64, workspace != nullptr);
  if (g.ws && (workspace_bytes < ws_bytes_of(g) || ((uintptr_t)workspace & 15) != 0)) g = plan_gemm(T, f, K, 64);
  if (!g.ws) (void)plan_pairs(T, f, K, 64, false, g);
  GemmParams p;
  p.y = (bf16*)y; p.bias = (const bf16*)bias_gate_up; p.T = T; p.N = f; p.K = K; p.act = 2; p.glu = glu; p.glu_alpha = glu_alpha; p.glu_limit = glu_limit;
  p.l2_hints = tunable(TUN_GEMM_L2_HINTS);
  p.trace = g_gemm_trace;
  p.ws_count = g.ws ? (unsigned int*)workspace : nullptr;
  p.ws_part = g.ws ? (float*)((uint8_t*)workspace + kWsCounterBytes) : nullptr;
  p.m_tiles = g.m_tiles; p.n_tiles = g.n_tiles; p.splits = g.splits;
  p.kb_total = g.kb_total; p.kb_per_split = g.kb_per_split; p.tokn = g.tokn;
  CUtensorMap tw, tx;
  if (int rc = make_tmap(&tw, w_gate_up, 2 * (int64_t)f, K, 64)) return rc;     // 64-row boxes: gate half, up half
  if (int rc = make_tmap(&tx, x, T, K, g.pair ? g.tokn / 2 : g.tokn)) return rc;
  return dispatch_gemm<true>(g, tw, tx, p, (cudaStream_t)stream);
}

extern "C" int KGE_GEMM_GATE_WS_NAME(void* y, const void* x, const void* w_gate_up, int T, int f, int K, void* workspace,
                                    int64_t workspace_bytes, void* stream) {
  return gemm_gated(y, x, w_gate_up, T, f, K, 0, 0.f, 0.f, workspace, workspace_bytes, stream);
}
extern "C" int KGE_GEMM_GLU_NAME(void* y, const void* x, const void* w_gate_up, int T, int f, int K, float alpha, float limit, void* workspace,
                                int64_t workspace_bytes, void* stream) {
  KGE_REQUIRE(limit > 0.f, "kge_gemm_clamped_glu_bf16: limit must be positive");
  return gemm_gated(y, x, w_gate_up, T, f, K, 1, alpha, limit, workspace, workspace_bytes, stream);
}

namespace kge {
inline namespace KGE_ELT_NS {
// the gated front half with biases: y[T, f] = silu(x w[:f]^T + b[:f]) * (x w[f:]^T + b[f:]), w [2f, K] and b [2f] stacked [gate | up]
int gemm_silu_gate_bias(void* y, const void* x, const void* w_gate_up, const void* bias_gate_up, int T, int f, int K, cudaStream_t st) {
  return gemm_gated(y, x, w_gate_up, T, f, K, 0, 0.f, 0.f, nullptr, 0, st, bias_gate_up);
}
// Grouped rows (the experts of a mixture, prompt steps): x [T, K] holds every group's rows padded to a multiple of 256,
// w stacks `groups` weight matrices ([N, K] each, or [2f, K] = [gate | up] with glu >= 0), tile_group (device, T / 256
// entries) names the matrix of every 256 rows.  y [T, N] (or [T, f]).  One launch for all groups, T > 256.
// glu: -1 plain projection, -2 plain projection followed by relu(.)^2, 0 silu(gate) * up, 1 the clamped pair.
int gemm_grouped(void* y, const void* x, const void* w, int T, int N, int K, int groups, const int32_t* tile_group, int glu, float glu_alpha,
                 float glu_limit, cudaStream_t st) {
  const bool gated = glu >= 0;
  KGE_REQUIRE(y && x && w && tile_group && groups > 0, "gemm_grouped: null pointer");
  KGE_REQUIRE(T > 256 && T % 256 == 0 && N > 0 && K > 0 && K % 8 == 0 && (!gated || N % 64 == 0), "gemm_grouped: T=%d N=%d K=%d", T, N, K);
  KGE_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0, "gemm_grouped: x and w must be 16-byte aligned");
  GemmPlan g = plan_gemm(T, N, K, gated ? 64 : BLK_M);
  (void)plan_pairs(T, N, K, gated ? 64 : BLK_M, true, g);
  KGE_REQUIRE(!g.ws && g.splits == 1 && 256 % g.tokn == 0, "gemm_grouped: internal: unexpected plan");
  GemmParams p;
  p.y = (bf16*)y; p.bias = nullptr; p.T = T; p.N = N; p.K = K; p.act = gated ? 2 : (glu == -2 ? 4 : 0);
  p.glu = gated ? glu : 0; p.glu_alpha = glu_alpha; p.glu_limit = glu_limit;
  p.l2_hints = tunable(TUN_GEMM_L2_HINTS); p.trace = g_gemm_trace; p.ws_count = nullptr; p.ws_part = nullptr;
  p.m_tiles = g.m_tiles; p.n_tiles = g.n_tiles; p.splits = g.splits; p.kb_total = g.kb_total; p.kb_per_split = g.kb_per_split; p.tokn = g.tokn;
  p.tile_group = tile_group; p.group_rows = gated ? 2 * N : N;
  CUtensorMap tw, tx;
  if (int rc = make_tmap(&tw, w, (int64_t)groups * p.group_rows, K, gated ? 64 : BLK_M)) return rc;
  if (int rc = make_tmap(&tx, x, T, K, g.pair ? g.tokn / 2 : g.tokn)) return rc;
  return gated ? dispatch_gemm<true>(g, tw, tx, p, st) : dispatch_gemm<false>(g, tw, tx, p, st);
}
}  // namespace KGE_ELT_NS
}  // namespace kge

extern "C" int KGE_GEMM_GATE_NAME(void* y, const void* x, const void* w_gate_up, int T, int f, int K, void* stream) {
  return KGE_GEMM_GATE_WS_NAME(y, x, w_gate_up, T, f, K, nullptr, 0, stream);
}
