// Prompt attention, two query tiles per CTA.  Included by attn_tc.cu inside its namespaces (tiles, descriptors, MMA wrappers).
//
// What bounds it: a 128 x 64 tile of scores costs 512 cycles of exponentials on an SM (16 a cycle) and 644 of the tensor pipe (S 8 x 48:
// an MMA of 64 keys waits for its operands from shared memory; P V 4 x 65).  A softmax warp that waits for its own chain (scores out of
// TMEM, maximum, exponentials, probabilities back) keeps neither busy, and one CTA's fill, drain and stores are not covered by another's
// work.  So one CTA per SM has
//   * two query tiles, each with four softmax warps (one row per thread) and an issuer of its own, so that neither waits for the other;
//     the second tile's exponentials start half a tile behind the first's (one handshake per item) and stay there: the stretches
//     without exponentials of one fall on the other's exponentials (4 x 2048 tokens: 136 -> 125 us)
//   * scores in one buffer and probabilities in two beside it (64 + 2 x 32 columns of TMEM): S of the next tile is issued as soon as the
//     scores are in registers.  (128-key tiles with P over S: 142 us, the softmax waited 1400 of 3200 cycles for P V and then S.)
//   * K and V tiles of 64 keys in rings of four, read by both query tiles, fetched by a warp of its own (block ids one box per lane)
//   * work handed out by the hardware's queue of CTAs not yet launched (clusterlaunchcontrol.try_cancel), asked for late, so that a
//     CTA goes on to the next item with its K, V and Q already on their way and long items do not wait behind each other
//   * an item that has one query tile only (single-token rows, short ends of prompts; all items of small launches) shares out its KEY
//     tiles between the two groups of warps, which merge at the end: half the serial walk of a decode row over its context
//   * outputs turned in shared memory so that rows leave in full lines (16 bytes of 32 rows per store took 3500 cycles an item).
// us before (128-row CTAs, two per SM) and now, 32 / 8 heads of 128: 4 x 2048 tokens 152 -> 125 (1097 TFLOP/s), one of 8192 467 -> 411
// (1337), 4 x 1000 61 -> 48, 37 decode rows of up to 3000 keys beside 2 x 1011 tokens behind 2777 181 -> 146, 200 decode rows beside 300
// tokens 128 -> 69.  Small launches stay with the other kernel (launch_tc).
namespace atc2 {
using namespace atc;

constexpr int kPairThreads = 384;              // warps 0-3 and 4-7: softmax of the first and second query tile; 8 and 9: their MMAs; 10: TMA
constexpr int kPairStages = 4;                 // K tiles and as many V tiles
template <int HD> constexpr int pair_smem() { return (2 * 128 + 2 * kPairStages * BNK) * HD * 2 + 512 + 8 * 4096 + 128 * 8; }

// n0, n1: key tiles of the two query tiles; n1 < 0: no more work.  split: there is one query tile, the even key tiles are the first
// one's and the odd ones the second one's.  tail: rows of the last tile that hold keys; 0: all of them, or the rest is zeros.
struct __align__(16) Item { int q0, tok0, ntok0, ntok1, ctx0, kvh, n0, n1, split, tile_lo, tail; };

// Outputs `ldo` apart and multiplied by out_scale.  BIAS kernels: a query at position i sees the keys j of its own chunk (chunk > 0; all up to i
// otherwise) with -slope (i - j) added to the scaled score, slope 2^(-span (head + 1) / H) (span > 0).  What is the same for a whole row drops
// out of the softmax but for the growth of its maximum, so distances are counted from the row's own position.
struct PairArgs { int ldo; float out_scale; int chunk; float span; };

__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
                 "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
template <int HD, bool BIAS>
__global__ void __launch_bounds__(kPairThreads, 1)
attn_pair_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_q8,
                 const __grid_constant__ CUtensorMap tm_q1, bf16* __restrict__ out, const bf16* __restrict__ k_cache, const bf16* __restrict__ v_cache,
                 const int32_t* __restrict__ block_table, int max_blocks,
                 const int32_t* __restrict__ seq_lens, const int32_t* __restrict__ qsl, int flat, int per, int H, int KV, int bs_shift, float scale_log2,
                 const float* __restrict__ sinks, const PairArgs pa) {
  constexpr int NST = kPairStages;
  constexpr uint32_t Q_TILE = 128 * HD * 2, TILE = BNK * HD * 2;
  // TMEM: O0 and O1, then per query tile the scores (64 columns) and two buffers of probabilities (32 columns each)
  constexpr uint32_t S_COL = 256;
  constexpr uint32_t IDESC_S = (1u << 4) | KGE_IDESC_AB | ((uint32_t)(BNK >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  constexpr uint32_t IDESC_O = (1u << 4) | KGE_IDESC_AB | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if ((s_addr(smem_raw) & 1023u) != 0) __trap();
  const uint32_t sQ = s_addr(smem_raw), sK = sQ + 2 * Q_TILE, sV = sK + NST * TILE;
  uint8_t* tail = smem_raw + 2 * Q_TILE + 2 * NST * TILE;
  const uint32_t bar0 = s_addr(tail);
  Item* items = reinterpret_cast<Item*>(tail + 288);                   // 2 slots of 48 bytes
  const uint32_t clc_resp = bar0 + 384;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 400);
  static_assert(sizeof(Item) == 48, "two items lie between the barriers and the answers to requests for work");
  // Barriers; tiles are counted over all items of the CTA.  A parity wait holds only while no later phase of its barrier can complete:
  // what completes the next phase needs something that the waiter does after the wait (p_full and o_full, which may run a tile ahead of
  // their waiters, are pairs for that).  No stage is handed back before it was filled: an issuer without work for a tile waits for it too.
  auto k_full = [&](int s) { return bar0 + 8u * s; };
  auto k_empty = [&](int s) { return bar0 + 32u + 8u * s; };
  auto v_full = [&](int s) { return bar0 + 64u + 8u * s; };
  auto v_empty = [&](int s) { return bar0 + 96u + 8u * s; };
  auto s_full = [&](int a) { return bar0 + 128u + 8u * a; };
  auto s_read = [&](int a) { return bar0 + 144u + 8u * a; };
  auto p_full = [&](int a, int t) { return bar0 + 160u + 16u * a + 8u * (t & 1); };
  auto o_full = [&](int a, int t) { return bar0 + 192u + 16u * a + 8u * (t & 1); };
  auto item_full = [&](int s) { return bar0 + 224u + 8u * s; };
  auto item_empty = [&](int s) { return bar0 + 240u + 8u * s; };
  const uint32_t q_full = bar0 + 256u, q_empty = bar0 + 264u, clc_full = bar0 + 272u;
  auto v_clean = [&](int s) { return bar0 + 408u + 8u * s; };
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int G = H / KV, TT = BM / G, TI = per * TT;     // tokens of a query tile, of an item

  if (warp == 8) {
    if (lane == 0) {
      for (int s = 0; s < NST; ++s) { mbar_init(k_full(s), 1); mbar_init(k_empty(s), 2); mbar_init(v_full(s), 1); mbar_init(v_empty(s), 2); mbar_init(v_clean(s), 1); }
      for (int a = 0; a < 2; ++a) {
        mbar_init(s_full(a), 1); mbar_init(s_read(a), 4);
        for (int t = 0; t < 2; ++t) { mbar_init(p_full(a, t), 4); mbar_init(o_full(a, t), 1); }
        mbar_init(item_full(a), 1); mbar_init(item_empty(a), 10);
      }
      mbar_init(q_full, 1); mbar_init(q_empty, 2); mbar_init(clc_full, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_addr(tmem_slot)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else if (warp == 10 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_v) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_q8) : "memory");
  }
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 10) {
    // ------------------------------------------------------------------ work items and TMA copies
    int bx = blockIdx.x, by = blockIdx.y, bz = blockIdx.z;
    const bool leader = elect_one();
    const int bs = 1 << bs_shift, box_rows = bs < BNK ? bs : BNK, boxes = BNK / box_rows;
    uint32_t nk = 0, ni = 0, nclc = 0;              // tiles, items and requests for work so far
    uint32_t gathered = 0;                          // barrier of the tile whose gathers are under way
    auto hand_over = [&](uint32_t next) {
      if (gathered) {
        if (next) cp_wait<1>(); else cp_wait<0>();
        fence_async_smem();
        __syncwarp();
        if (leader) mbar_arrive(gathered);
      }
      gathered = next;
    };
    while (true) {
      int rank = bz, kvh = bx, b = by;
      if (flat) {
        // work number bx / KV in the requests' order from the last to the first, without gaps: 32 requests at a time
        kvh = bx % KV;
        rank = bx / KV;
        for (b = -1; b < 0;) {
          const int r = by + lane, mine = r < flat ? (qsl[flat - r] - qsl[flat - 1 - r] + TI - 1) / TI : 0;
          int upto = mine;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
          }
          const uint32_t past = __ballot_sync(0xffffffffu, upto > rank);
          if (past) {
            const int l = __ffs(past) - 1;
            rank -= __shfl_sync(0xffffffffu, upto - mine, l);
            b = flat - 1 - by - l;
          } else {
            rank -= __shfl_sync(0xffffffffu, upto, 31);
            by += 32;
            if (by >= flat) { b = 0; rank = -1; }                      // more CTAs than work
          }
        }
      }
      // everything that the first copies need is asked for at once: lengths, and the ids of the first 32 boxes, one per lane
      const int32_t* btab = block_table + (int64_t)b * max_blocks;
      const int q0 = qsl[b], q1 = qsl[b + 1], seq_len = seq_lens[b], id0 = btab[min((lane * box_rows) >> bs_shift, max_blocks - 1)];
      const int q_len = q1 - q0;
      const int tok0 = rank < 0 ? -1 : ((q_len + TI - 1) / TI - 1 - rank) * TI;
      if (tok0 >= 0) {
        const int ctx0 = seq_len - q_len;
        const int ntok0 = min(TT, q_len - tok0), ntok1 = max(0, min(TI - TT, q_len - tok0 - TT));
        const int kv_len = ctx0 + tok0 + ntok0 + ntok1;
        const int tile_lo = BIAS && pa.chunk > 0 ? (ctx0 + tok0) / pa.chunk * pa.chunk / BNK : 0;      // where the first query's chunk begins
        const int n = (kv_len + BNK - 1) / BNK - tile_lo, split = ntok1 == 0 && n > 1;
        const int n0 = split ? (n + 1) / 2 : (ctx0 + tok0 + ntok0 + BNK - 1) / BNK - tile_lo, n1 = split ? n / 2 : (ntok1 ? n : 0);
        const int slot = ni & 1;
        if (ni >= 2) mbar_wait(item_empty(slot), ((ni >> 1) - 1) & 1);
        if (leader) {
          Item it;
          it.q0 = q0; it.tok0 = tok0; it.ntok0 = ntok0; it.ntok1 = ntok1; it.ctx0 = ctx0; it.kvh = kvh; it.n0 = n0; it.n1 = n1; it.split = split; it.tile_lo = tile_lo; it.tail = k_cache ? 0 : kv_len % BNK;
          items[slot] = it;
          mbar_arrive(item_full(slot));
        }
        __syncwarp();
        // block ids of 32 boxes at a time; a box beyond the keys repeats the block of the first key (its scores are masked)
        int ids_at = 0, ids = lane * box_rows < kv_len ? id0 : -1;
        const int block0 = __shfl_sync(0xffffffffu, id0, 0);
        if (ids < 0) ids = block0;
        auto fetch = [&](int j, bool is_k) {
          const int st = nk % NST;
          if (nk >= (uint32_t)NST) mbar_wait(is_k ? k_empty(st) : v_empty(st), (nk / NST - 1) & 1);
          const uint32_t dst = (is_k ? sK : sV) + st * TILE, bar = is_k ? k_full(st) : v_full(st);
          if (leader && !k_cache) mbar_expect_tx(bar, TILE);
          const int first = j * boxes;
          if (ids_at != first / 32) {
            ids_at = first / 32;
            const int key = (ids_at * 32 + lane) * box_rows;
            ids = key < kv_len ? btab[min(key >> bs_shift, max_blocks - 1)] : block0;
          }
          if (k_cache) {
            // knob "attn_tma" 0: the same tiles gathered by the lanes (zeros beyond the keys); a tile is handed over when the next one's
            // copies are under way
            constexpr int CH = HD / 8;
#pragma unroll 4
            for (int i = lane; i < BNK * CH; i += 32) {
              const int row = i / CH, chunk = i % CH;
              const int blk = __shfl_sync(0xffffffffu, ids, (first + row / box_rows) & 31);
              const bf16* src = (is_k ? k_cache : v_cache) + ((int64_t)(blk * KV + kvh) * bs + ((j * BNK + row) & (bs - 1))) * HD + chunk * 8;
              cp16(dst + tile_off<BNK>(row, chunk), src, j * BNK + row < kv_len);
            }
            cp_commit();
            hand_over(bar);
            return;
          }
          for (int i = 0; i < boxes; ++i) {
            const int blk = __shfl_sync(0xffffffffu, ids, (first + i) & 31);
            const int row = (blk * KV + kvh) * bs + ((j * BNK + i * box_rows) & (bs - 1));
            if (leader) {
#pragma unroll
              for (int h = 0; h < HD / 64; ++h)
                tma_load_2d(dst + (uint32_t)(h * (BNK * 128) + i * box_rows * 128), is_k ? &tm_k : &tm_v, bar, h * 64, row);
            }
          }
        };
        // Q: boxes of 8 tokens, single tokens for the rest, so that nothing beyond the request's rows is read
        if (ni > 0) mbar_wait(q_empty, (ni - 1) & 1);
        if (leader) {
          mbar_expect_tx(q_full, (uint32_t)((ntok0 + ntok1) * G * HD * 2));
#pragma unroll 1
          for (int a = 0; a < 2; ++a) {
            const int nt = a ? ntok1 : ntok0, full = TT >= 8 ? nt & ~7 : 0;
            for (int t = 0; t < nt; t += t < full ? 8 : 1)
#pragma unroll
              for (int h = 0; h < HD / 64; ++h)
                tma_load_3d(sQ + a * Q_TILE + (uint32_t)(h * (128 * 128) + t * G * 128), t < full ? &tm_q8 : &tm_q1, q_full, h * 64, kvh * G, q0 + tok0 + a * TT + t);
          }
        }
        __syncwarp();
        for (int j = 0; j < n; ++j) {
          fetch(tile_lo + j, true);
          fetch(tile_lo + j, false);
          ++nk;
        }
        hand_over(0);
        ++ni;
      }
      // the next item is asked for with the last tiles of this one in flight: asked for earlier, it would be tied to a CTA that is still
      // long busy (256 items of one prompt: 57 us when each CTA asked at an item's start)
      if (leader) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(clc_full, 16);
        asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(clc_resp), "r"(clc_full) : "memory");
      }
      __syncwarp();
      mbar_wait(clc_full, nclc & 1);
      ++nclc;
      uint32_t ok, x = 0, y = 0, z = 0;
      asm volatile(
          "{\n.reg .b128 h;\n.reg .pred p;\nld.shared.b128 h, [%4];\n"
          "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\nselp.u32 %0, 1, 0, p;\n"
          "mov.b32 %1, 0;\nmov.b32 %2, 0;\nmov.b32 %3, 0;\n"
          "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, h;\n}"
          : "=r"(ok), "=r"(x), "=r"(y), "=r"(z) : "r"(clc_resp) : "memory");
      __syncwarp();
      if (!ok) break;
      bx = (int)x; by = (int)y; bz = (int)z;
    }
    const int slot = ni & 1;
    if (ni >= 2) mbar_wait(item_empty(slot), ((ni >> 1) - 1) & 1);
    if (leader) {
      items[slot].n1 = -1;
      mbar_arrive(item_full(slot));
    }
  } else if (warp == 8 || warp == 9) {
    // ------------------------------------------------------------------ MMA issuer of query tile a
    if (elect_one()) {
      const int a = warp - 8;
      const uint32_t t_s = tmem + S_COL + a * 128, t_o = tmem + a * 128;
      uint32_t ns = 0, np = 0, nk = 0;                 // score tiles and products P V issued so far, key tiles
      uint32_t cleaned = 0;                            // parities of the stages' next v_clean
      for (uint32_t ni = 0;; ++ni) {
        mbar_wait(item_full(ni & 1), (ni >> 1) & 1);
        const int n0 = items[ni & 1].n0, n1 = items[ni & 1].n1, split = items[ni & 1].split, tail = items[ni & 1].tail;
        mbar_arrive(item_empty(ni & 1));
        if (n1 < 0) break;
        const bool shared_tail = !split && n0 == n1;   // both query tiles see the last key tile
        const int n = split ? n0 + n1 : max(n0, n1), na = a ? n1 : n0, ahead = 1 + split;
        const uint64_t qd = desc_kmajor(sQ + (split ? 0 : a) * Q_TILE);
        mbar_wait(q_full, ni & 1);
        bool first = true;                             // no product P V of this item yet
        for (int j = -ahead; j < n; ++j) {
          const int js = j + ahead;
          if (js < n) {                                // S of a tile ahead, once the softmax has read the one before
            const int st = (nk + js) % NST;
            mbar_wait(k_full(st), ((nk + js) / NST) & 1);         // also without work for it: the stage is not handed back before it is filled
            if (split ? (js & 1) == a : js < na) {
              if (ns > 0) mbar_wait(s_read(a), (ns - 1) & 1);
              tc_after();
              const uint64_t kd = desc_kmajor(sK + st * TILE);
#pragma unroll
              for (int k = 0; k < HD / 16; ++k) {
                const uint32_t qoff = (uint32_t)((k >> 2) * (128 * 128) + (k & 3) * 32), koff = (uint32_t)((k >> 2) * (BNK * 128) + (k & 3) * 32);
                tc_mma(t_s, qd + (qoff >> 4), kd + (koff >> 4), IDESC_S, k > 0 ? 1u : 0u);
              }
              tc_commit(s_full(a));
              ++ns;
            }
            tc_commit(k_empty(st));
            if (js + 1 == n) tc_commit(q_empty);
          }
          if (j >= 0) {                                // P V of tile j
            const int st = (nk + j) % NST;
            mbar_wait(v_full(st), ((nk + j) / NST) & 1);
            if (split ? (j & 1) == a : j < na) {
              // values beyond the last key (clean_tail), by one issuer where both use the tile.  (Cleared before the tile is handed over, by the
              // producer or a warp of its own, 200 decode rows beside 300 tokens took 126 us, 119.8 here and 121.0 without.)
              int groups = BNK / 16;
              if (tail && j + 1 == n) {
                if (shared_tail && a == 1) {
                  mbar_wait(v_clean(st), (cleaned >> st) & 1);
                  cleaned ^= 1u << st;
                  groups = (tail + 15) / 16;
                } else {
                  groups = clean_tail<HD>(sV + st * TILE, tail);
                  if (shared_tail) mbar_arrive(v_clean(st));
                }
              }
              mbar_wait(p_full(a, np), (np >> 1) & 1);
              tc_after();
              const uint64_t vd = desc_mnmajor(sV + st * TILE);
              const uint32_t t_p = t_s + 64 + (np & 1) * 32;
#pragma unroll
              for (int k = 0; k < BNK / 16; ++k)
                if (k < groups)
                  tc_mma_ts(t_o, t_p + k * 8, vd + (uint32_t)((k * 16 * 128) >> 4), IDESC_O, (!first || k > 0) ? 1u : 0u);
              tc_commit(o_full(a, np));
              ++np;
              first = false;
            }
            tc_commit(v_empty(st));
          }
        }
        nk += n;
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ softmax: one row per thread
    const int a = warp >> 2, r = threadIdx.x & 127, tk = r / G, hh = r % G;
    const uint32_t t_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t t_s = t_row + S_COL + a * 128, t_o = t_row + a * 128;
    const f2 sc2 = pk(scale_log2, scale_log2);
    uint32_t ns = 0;
    for (uint32_t ni = 0;; ++ni) {
      mbar_wait(item_full(ni & 1), (ni >> 1) & 1);
      const Item it = items[ni & 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(item_empty(ni & 1));
      if (it.n1 < 0) break;
      const int n = a ? it.n1 : it.n0;
      if (n <= 0) continue;
      const int qt = it.split ? 0 : a;                                 // the query tile of these warps
      const bool row_ok = tk < (qt ? it.ntok1 : it.ntok0);
      const int row_tok = it.tok0 + qt * TT + tk;
      const int lim = row_ok ? it.ctx0 + row_tok : -1;                 // last visible key of this row
      const int head = it.kvh * G + hh;
      const int lo_row = BIAS && row_ok && pa.chunk > 0 ? lim / pa.chunk * pa.chunk : 0;      // its first key
      const float slope2 = BIAS && pa.span > 0.f ? exp2f(-pa.span * (float)(head + 1) / (float)H) * kLog2e : 0.f;
      float m_ref = -INFINITY, l = 0.f;
      // the second group's exponentials start when the first's of its first tile are done.  From three tiles of the second group on: then
      // the first group cannot come to its next item's handshake before the second has passed this one (it needs Q, which waits for the
      // second group's last scores to be issued, and those for its second tile to be read)
      const bool turns = it.n1 >= 3;
      for (int j = 0; j < n; ++j) {
        mbar_wait(s_full(a), ns & 1);
        tc_after();
        uint32_t sv[BNK];
#pragma unroll
        for (int c = 0; c < BNK; c += 32) tmem_ld32_nowait(t_s + c, &sv[c]);
        tmem_wait_ld(sv);
        tc_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_read(a));                         // the next tile's scores may be written
        const int kbase = (it.tile_lo + (it.split ? 2 * j + a : j)) * BNK, vis = lim - kbase, from = lo_row - kbase;      // columns from .. vis are visible
        float mxa[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (BIAS) {
          const f2 sl2 = pk(slope2, slope2), b2 = pk(-slope2 * (float)vis, -slope2 * (float)vis);
#pragma unroll
          for (int i = 0; i < BNK; i += 2) {
            float x0, x1;
            upk(fma2(pk(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sc2, fma2(pk((float)i, (float)(i + 1)), sl2, b2)), x0, x1);
            sv[i] = __float_as_uint(x0); sv[i + 1] = __float_as_uint(x1);
          }
        }
        if (!__all_sync(0xffffffffu, vis >= BNK - 1 && (!BIAS || from <= 0))) {
#pragma unroll
          for (int i = 0; i < BNK; ++i) sv[i] = i <= vis && (!BIAS || i >= from) ? sv[i] : 0xff800000u;
        }
#pragma unroll
        for (int i = 0; i < BNK; i += 8)
#pragma unroll
          for (int k = 0; k < 4; ++k) mxa[k] = max3(mxa[k], __uint_as_float(sv[i + 2 * k]), __uint_as_float(sv[i + 2 * k + 1]));
        const float mx = max3(fmaxf(mxa[0], mxa[1]), mxa[2], mxa[3]) * (BIAS ? 1.f : scale_log2);      // -inf stays -inf
        // includes the first finite maximum.  BIAS: any growth, so that a row's largest weight is one and is not rounded, as in the kernel that
        // had these prompts (a reference up to 2^8 behind: error up to 6 % larger, 0.00174 against 0.00165 at 700 keys, and no faster)
        const bool grow = mx > m_ref + (BIAS ? 0.f : kRescaleThreshold);
        if (__any_sync(0xffffffffu, grow)) {
          float alpha = 1.f;
          if (grow) {
            alpha = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - mx);
            m_ref = mx;
            l *= alpha;
          }
          if (j > 0) {
            mbar_wait(o_full(a, ns - 1), ((ns - 1) >> 1) & 1);         // P V of the tile before
            tc_after();
#pragma unroll 1
            for (int c = 0; c < HD; c += 16) {
              uint32_t v[16];
              asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                           : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                             "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(t_o + c));
              tmem_wait_ld(v);
#pragma unroll
              for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
              tmem_st16(t_o + c, v);
            }
          }
        }
        const float base = (m_ref == -INFINITY) ? 0.f : m_ref;
        const f2 nb2 = pk(-base, -base);
        f2 rs[2] = {0, 0};
        if (ns >= 2) { mbar_wait(o_full(a, ns), ((ns - 2) >> 1) & 1); tc_after(); }       // P V of two tiles before has read this buffer
        if (turns && j == 0 && a == 1) asm volatile("bar.sync 1, 256;" ::: "memory");
        const uint32_t t_p = t_s + 64 + (ns & 1) * 32;
#pragma unroll
        for (int c = 0; c < BNK; c += 32) {
          uint32_t pkd[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float p0, p1;
            const f2 x = pk(__uint_as_float(sv[c + 2 * i]), __uint_as_float(sv[c + 2 * i + 1]));
            upk(BIAS ? add2(x, nb2) : fma2(x, sc2, nb2), p0, p1);
            p0 = ex2_ftz(p0); p1 = ex2_ftz(p1);                        // masked: -inf -> 0
            rs[i & 1] = add2(rs[i & 1], pk(p0, p1));
            pkd[i] = pack_bf2(p0, p1);
          }
          tmem_st16(t_p + c / 2, pkd);
        }
        if (turns && j == 0 && a == 0) asm volatile("bar.arrive 1, 256;" ::: "memory");
        tmem_wait_st();
        tc_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full(a, ns));
        ++ns;
        l += sum2(add2(rs[0], rs[1]));
      }
      mbar_wait(o_full(a, ns - 1), ((ns - 1) >> 1) & 1);
      tc_after();
      float2* part = reinterpret_cast<float2*>(smem_raw + 2 * Q_TILE + 2 * NST * TILE + 512 + 8 * 4096);
      float mine = 1.f, other = 0.f;                                   // weights of the two halves of a split row
      if (it.split) {
        // the second half's warps hand over their sums; their P V is done, and O1 is read by the first half's (a warp reads the TMEM
        // lanes of its number mod 4, whichever columns)
        if (a) part[r] = make_float2(m_ref, l);
        tc_before();
        asm volatile("bar.sync 2, 256;" ::: "memory");
        tc_after();
        if (!a) {
          const float2 p1 = part[r];
          const float m = fmaxf(m_ref, p1.x);
          mine = m_ref == -INFINITY ? 0.f : exp2f(m_ref - m);
          other = p1.x == -INFINITY ? 0.f : exp2f(p1.x - m);
          l = l * mine + p1.y * other;
          m_ref = m;
        }
      }
      if (sinks && row_ok && m_ref != -INFINITY) l += exp2f(sinks[head] * kLog2e - m_ref);
      const float inv = l > 0.f ? pa.out_scale / l : 0.f;
      // a warp turns its 32 rows in shared memory, 64 columns at a time, and stores 128 contiguous bytes of four rows at once (16 bytes
      // of each row by its own thread: a third of the time of a short item)
      uint8_t* stage = smem_raw + 2 * Q_TILE + 2 * NST * TILE + 512 + warp * 4096;
      const int srow = lane >> 3, schunk = lane & 7;
      const uint32_t rows_ok = __ballot_sync(0xffffffffu, row_ok);
#pragma unroll 1
      for (int c = 0; c < HD && !(it.split && a); c += 64) {
        uint32_t v[64];
        tmem_ld32_nowait(t_o + c, v);
        tmem_ld32_nowait(t_o + c + 32, v + 32);
        tmem_wait_ld(v);
        if (it.split) {
#pragma unroll
          for (int h = 0; h < 64; h += 32) {
            uint32_t u[32];
            tmem_ld32_nowait(t_o + 128 + c + h, u);
            tmem_wait_ld(u);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[h + i] = __float_as_uint(__uint_as_float(v[h + i]) * mine + __uint_as_float(u[i]) * other);
          }
        }
        tc_before();                                                   // the next item's first P V comes behind p_full of these warps
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 64; i += 8) {
          uint4 w;
          w.x = pack_bf2(__uint_as_float(v[i]) * inv, __uint_as_float(v[i + 1]) * inv);
          w.y = pack_bf2(__uint_as_float(v[i + 2]) * inv, __uint_as_float(v[i + 3]) * inv);
          w.z = pack_bf2(__uint_as_float(v[i + 4]) * inv, __uint_as_float(v[i + 5]) * inv);
          w.w = pack_bf2(__uint_as_float(v[i + 6]) * inv, __uint_as_float(v[i + 7]) * inv);
          *reinterpret_cast<uint4*>(stage + lane * 128 + (((i >> 3) ^ (lane & 7)) << 4)) = w;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const int row = i + srow, rr = (warp & 3) * 32 + row, t2 = rr / G;
          const uint4 w = *reinterpret_cast<const uint4*>(stage + row * 128 + ((schunk ^ (row & 7)) << 4));
          if ((rows_ok >> row) & 1)
            *reinterpret_cast<uint4*>(out + (int64_t)(it.q0 + it.tok0 + qt * TT + t2) * pa.ldo + (it.kvh * G + rr - t2 * G) * HD + c + schunk * 8) = w;
        }
      }
      if (it.split) {                                                  // O1 and the sums are read
        asm volatile("bar.sync 3, 256;" ::: "memory");
      }
    }
  }
  tc_before();
  __syncthreads();
  if (warp == 8) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
}
}  // namespace atc2

int make_tmap(CUtensorMap* m, const void* ptr, int64_t rows, int64_t cols, int box_rows);   // gemm_tc.cu (cached)
int make_tmap_q(CUtensorMap* m, const void* ptr, int64_t stride, int hd, int heads, int box_heads, int box_tokens);     // gemm_tc.cu (cached)

template <int HD, bool BIAS>
static int launch_pair(const atc2::PairArgs& pa, bf16* out, const bf16* q, int q_stride, const bf16* kc, const bf16* vc, const int32_t* bt, int max_blocks, const int32_t* sl,
                       const int32_t* qsl, int B, int T, int max_q_len, int max_seq_len, int H, int KV, int bs, int bs_shift, float scale, const float* sinks, cudaStream_t st) {
  const int G = H / KV, TT = atc::BM / G, box_rows = bs < atc::BNK ? bs : atc::BNK;
  // Query tiles per item: two, sharing the K and V tiles (us with two / one and its key tiles split: 4 x 2048 tokens 125 / 169, two of
  // 1024 26.7 / 35), unless that leaves SMs without an item or with one long one (one of 512 15.7 / 11.3, one of 1024 20.5 / 18.2,
  // 2 x 4000 with 4 / 4 heads 69 / 43; but 8 x 128 11.4 / 12.3, two of 400 11.9 / 13.0).
  int by_request = 0, per = 2;
  dim3 grid = tc_grid(B, T, max_q_len, per * TT, KV, by_request);
  auto items = [&] { return by_request ? KV * ((int64_t)T / (per * TT) + B) : (int64_t)grid.x * grid.y * grid.z; };
  if (items() <= 74 || (items() <= 148 && max_seq_len >= 512)) {
    per = 1;
    grid = tc_grid(B, T, max_q_len, per * TT, KV, by_request);
  }
  if (by_request) grid = dim3((unsigned)items());
  CUtensorMap tk, tv, tq8, tq1;
  const bf16 *gk = nullptr, *gv = nullptr;
  const int64_t rows = (int64_t)1 << 30;
  if (int rc = make_tmap(&tk, kc, rows, HD, box_rows)) return rc;
  if (int rc = make_tmap(&tv, vc, rows, HD, box_rows)) return rc;
  if (int rc = make_tmap_q(&tq1, q, q_stride, HD, H, G, 1)) return rc;
  tq8 = tq1;
  if (TT >= 8) { if (int rc = make_tmap_q(&tq8, q, q_stride, HD, H, G, 8)) return rc; }
  if (!tunable(TUN_ATTN_TMA)) { gk = kc; gv = vc; }
  auto kern = atc2::attn_pair_kernel<HD, BIAS>;
  KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, atc2::pair_smem<HD>()));
  KGE_CUDA_OK(launch_pdl(kern, grid, dim3(atc2::kPairThreads), atc2::pair_smem<HD>(), st, tk, tv, tq8, tq1, out, gk, gv, bt, max_blocks, sl, qsl, by_request ? B : 0, per, H, KV,
                         bs_shift, scale * atc::kLog2e, sinks, pa));
  return 0;
}
