// Projections of a few token rows (T <= 16): y[T,N] = act(x[T,K] * w[N,K]^T + bias), plain or gated.  Included by gemm_tc.cu
// inside its namespaces (GemmParams, apply_act, silu_gate_bf16).
//
// Every weight is used T times at most, so the job is to get the weights through the SMs once and quickly; at the sizes where
// this kernel is chosen a launch lasts a few microseconds and what costs is latency: of a TMA ring filling, of TMEM being
// allocated, of an MMA chain, of a cluster exchange.  Here a warp streams its own weights: mma.m16n8k16 with the tokens as its
// 16 rows and 8 weight rows as its columns, and since the order of a contraction is free, lane t of a quad takes 16 consecutive
// bytes (8 numbers of k) of each 32-number piece of both operands, which feeds two MMAs.  A lane copies its pieces by cp.async
// into shared memory and reads back only what it copied, so there is no barrier in the main loop; the first stages of weights
// are requested before the previous kernel has finished.  (Loads straight into registers had 3.2 TB/s at most: with the L1 split
// that all kernels ask for, what L1 can hold bounds the loads in flight.)  The warps of a CTA interleave over K in chunks of 64
// and add their sums in shared memory in warp order (the same bits in every run).
// Back-to-back launches on cold weights, us at 1 token (the TMA kernels in brackets): 768 x 768 1.6 (3.6), 3072 x 768 2.0 (3.9),
// 768 x 3072 2.2 (4.1), 2048 x 2048 3.2 (4.8), 4096 x 4096 6.9 (9.2), 16384 x 2048 gated 14.2 (16.4), 28672 x 4096 gated 42.3 (46.5),
// 4096 x 14336 20.2 (21.4), 5.8 TB/s.
constexpr int kRowsMaxT = 16;

__device__ __forceinline__ void rows_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32." KGE_MMA_ELT "." KGE_MMA_ELT ".f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int rows_smem(int warps, int nw, int tt, int s) { return warps * s * (nw + tt) * 1024; }

// NORM: the rows are normalised first, each by one warp, in every CTA (a row of 768 is 1.5 KB from L2; a kernel of its own costs the
// latency of one more launch in the chain of a step); their 16-bit values lie in shared memory behind the ring.
constexpr int kNormVecs = 4;                           // 16-byte pieces of a row per lane: up to 1024 of K
__host__ __device__ constexpr int norm_row_bytes(int K) { return 2 * K + 64; }      // the fragments of eight rows fall on different banks

__device__ __forceinline__ void unpack8(uint4 a, float (&f)[8]) {
  f[0] = bf_lo(a.x); f[1] = bf_hi(a.x); f[2] = bf_lo(a.y); f[3] = bf_hi(a.y);
  f[4] = bf_lo(a.z); f[5] = bf_hi(a.z); f[6] = bf_lo(a.w); f[7] = bf_hi(a.w);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf2(f[0], f[1]), pack_bf2(f[2], f[3]), pack_bf2(f[4], f[5]), pack_bf2(f[6], f[7]));
}

__device__ __forceinline__ void norm_weights(uint4 (&wv)[kNormVecs], uint4 (&bv)[kNormVecs], const RowsNorm& nm, int K) {
#pragma unroll
  for (int j = 0; j < kNormVecs; ++j) {
    const int i = (threadIdx.x & 31) + j * 32;
    if (i < K / 8) {
      wv[j] = *reinterpret_cast<const uint4*>((const bf16*)nm.w + i * 8);
      bv[j] = *reinterpret_cast<const uint4*>((const bf16*)nm.b + i * 8);
    }
  }
}
// One row by one warp, with the roundings of norm_kernel (elementwise.cu)
__device__ __forceinline__ void norm_row(uint8_t* dst, const RowsNorm& nm, const uint4 (&wv)[kNormVecs], const uint4 (&bv)[kNormVecs], int row, int K, bool store) {
  const int lane = threadIdx.x & 31, nvec = K / 8;
  const int64_t base = (int64_t)row * K;
  const bf16 *res = (const bf16*)nm.res + base, *add = (const bf16*)nm.add + base;
  // every load before the first store: behind a store to res_out the compiler keeps later loads back, and each costs a trip to L2
  uint4 rv[kNormVecs], av[kNormVecs];
#pragma unroll
  for (int j = 0; j < kNormVecs; ++j) {
    const int i = lane + j * 32;
    if (i < nvec) {
      rv[j] = *reinterpret_cast<const uint4*>(res + i * 8);
      if (nm.add) av[j] = *reinterpret_cast<const uint4*>(add + i * 8);
    }
  }
  float v[kNormVecs][8], acc = 0.f;
#pragma unroll
  for (int j = 0; j < kNormVecs; ++j) {
    const int i = lane + j * 32;
    if (i < nvec) {
      unpack8(rv[j], v[j]);
      if (nm.add) {
        float r[8];
        unpack8(av[j], r);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j][k] += r[k];
        const uint4 o = pack8(v[j]);
        if (store) *reinterpret_cast<uint4*>((bf16*)nm.res_out + base + i * 8) = o;
        unpack8(o, v[j]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) acc += v[j][k];
    }
  }
  const float mean = warp_sum(acc) / (float)K;
  float a2 = 0.f;
#pragma unroll
  for (int j = 0; j < kNormVecs; ++j)
    if (lane + j * 32 < nvec)
#pragma unroll
      for (int k = 0; k < 8; ++k) { const float c = v[j][k] - mean; a2 += c * c; }
  const float rstd = 1.0f / sqrtf(warp_sum(a2) / (float)K + nm.eps);
#pragma unroll
  for (int j = 0; j < kNormVecs; ++j) {
    const int i = lane + j * 32;
    if (i < nvec) {
      float wf[8], bf[8], o[8];
      unpack8(wv[j], wf);
      unpack8(bv[j], bf);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = (v[j][k] - mean) * rstd * wf[k] + bf[k];
      *reinterpret_cast<uint4*>(dst + i * 16) = pack8(o);
    }
  }
}

// W: warps per CTA; NT: 8-row weight tiles per CTA (GATED: NT of gate rows and NT of their up rows); TT: 8-token halves in
// use; S: stages of 64 of K per warp
template <int W, int NT, int TT, bool GATED, int S, bool NORM = false>
__global__ void __launch_bounds__(W * 32, NORM ? 2 : 1)
gemm_rows_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, const GemmParams p, const RowsNorm nm, const RowsKv kv) {
  static_assert(!NORM || TT == 1, "up to 8 normalised rows");
  constexpr int NW = GATED ? 2 * NT : NT, PIECES = 2 * (NW + (NORM ? 0 : TT));
  extern __shared__ __align__(16) uint4 ring[];        // [warp][stage][piece][lane]
  __shared__ float part[W][TT * 8][NW * 8 + 2];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * (8 * NT), chunks = (p.K + 63) / 64;
  const int mine = chunks > warp ? (chunks - warp + W - 1) / W : 0;
  const bf16* wrow[NW];
#pragma unroll
  for (int j = 0; j < NW; ++j) {
    const int n = min(n0 + (j % NT) * 8 + g, p.N - 1) + (j >= NT ? p.N : 0);       // a column beyond N is not stored
    wrow[j] = w + (int64_t)n * p.K + t * 8;
  }
  const bf16* xrow = x + (int64_t)g * p.K + t * 8;
  uint4* slot0 = ring + (warp * S * PIECES) * 32 + lane;
  auto copy = [&](uint4* dst, const bf16* src, bool in) {
    const uint32_t bytes = in ? 16u : 0u;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(in ? src : w), "r"(bytes) : "memory");
  };
  auto copy_w = [&](int i) {                           // chunk number i of this warp
    uint4* dst = slot0 + (i % S) * PIECES * 32;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = (warp + i * W) * 64 + h * 32;
#pragma unroll
      for (int j = 0; j < NW; ++j) copy(dst + (2 * j + h) * 32, wrow[j] + k, k + t * 8 < p.K);
    }
  };
  auto copy_x = [&](int i) {
    uint4* dst = slot0 + ((i % S) * PIECES + 2 * NW) * 32;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = (warp + i * W) * 64 + h * 32;
#pragma unroll
      for (int j = 0; j < TT; ++j) copy(dst + (2 * j + h) * 32, xrow + (int64_t)(8 * j) * p.K + k, k + t * 8 < p.K && g + 8 * j < p.T);
    }
  };
  float acc[NW][4];
#pragma unroll
  for (int j = 0; j < NW; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

#pragma unroll
  for (int i = 0; i < S - 1; ++i)
    if (i < mine) copy_w(i);
  uint4 nw[kNormVecs], nb[kNormVecs];
  if (NORM && warp < p.T) norm_weights(nw, nb, nm, p.K);
  // the bias of this thread's first output: a trip to memory behind the sums otherwise
  const int first_n = n0 + (int)threadIdx.x % (8 * NT);
  const float first_bias = !GATED && p.bias && first_n < p.N ? bf2f(p.bias[first_n]) : 0.f;
  pdl_wait();                                          // the tokens are the previous kernel's output
#pragma unroll
  for (int i = 0; i < S - 1; ++i) {
    if (!NORM && i < mine) copy_x(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  uint8_t* rows = reinterpret_cast<uint8_t*>(ring + W * S * PIECES * 32);
  const uint8_t* my_row = rows + min(g, p.T - 1) * norm_row_bytes(p.K) + t * 16;      // what rows beyond T hold is not stored
  if (NORM) {
    if (warp < p.T) norm_row(rows + warp * norm_row_bytes(p.K), nm, nw, nb, warp, p.K, blockIdx.x == 0);
    __syncthreads();
  }
#pragma unroll 1
  for (int i = 0; i < mine; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    const uint4* src = slot0 + (i % S) * PIECES * 32;
    uint4 wv[NW][2], xv[TT][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int j = 0; j < NW; ++j) wv[j][h] = src[(2 * j + h) * 32];
      if (NORM) {
        const int k = (warp + i * W) * 64 + h * 32;
        xv[0][h] = k + t * 8 < p.K ? *reinterpret_cast<const uint4*>(my_row + 2 * k) : make_uint4(0, 0, 0, 0);
      } else {
#pragma unroll
        for (int j = 0; j < TT; ++j) xv[j][h] = src[(2 * (NW + j) + h) * 32];
      }
    }
    if (i + S - 1 < mine) {                            // into the stage that the previous turn read
      copy_w(i + S - 1);
      if (!NORM) copy_x(i + S - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 lo = xv[0][h], hi = TT > 1 ? xv[TT - 1][h] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < NW; ++j) {
        rows_mma(acc[j], lo.x, hi.x, lo.y, hi.y, wv[j][h].x, wv[j][h].y);
        rows_mma(acc[j], lo.z, hi.z, lo.w, hi.w, wv[j][h].z, wv[j][h].w);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < NW; ++j)
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) part[warp][i * 8 + g][j * 8 + t * 2 + q] = acc[j][2 * i + q];
  __syncthreads();
  // one output per thread and trip, consecutive columns in consecutive threads
  for (int i = threadIdx.x; i < p.T * 8 * NT; i += W * 32) {
    const int tok = i / (8 * NT), col = i % (8 * NT), n = n0 + col;
    if (n >= p.N) continue;
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int s = 0; s < W; ++s) {
      a += part[s][tok][col];
      if (GATED) b += part[s][tok][NT * 8 + col];
    }
    float v;
    if (GATED) v = silu_gate_bf16(p, a, b, n);
    else v = apply_act(p.bias ? a + first_bias : a, p.act);             // W * 32 is a multiple of 8 NT: every trip has the same column
    p.y[(int64_t)tok * p.N + n] = f2bf(v);
    if (NORM && kv.kc && n >= kv.q_cols) {             // a key or a value: into the cache too
      const int64_t slot = kv.slots[tok];
      const int c = n - kv.q_cols, width = kv.KV * kv.hd, u = c < width ? c : c - width;
      if (slot >= 0)
        (c < width ? (bf16*)kv.kc : (bf16*)kv.vc)[(((slot / kv.bs) * kv.KV + u / kv.hd) * kv.bs + slot % kv.bs) * kv.hd + u % kv.hd] = f2bf(v);
    }
  }
}

template <int W, int NT, int TT, bool GATED, int S>
static int launch_rows_as(const bf16* x, const bf16* w, const GemmParams& p, cudaStream_t st) {
  auto kern = gemm_rows_kernel<W, NT, TT, GATED, S>;
  constexpr int smem = rows_smem(W, GATED ? 2 * NT : NT, TT, S);
  KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  KGE_CUDA_OK(launch_pdl(kern, dim3((p.N + 8 * NT - 1) / (8 * NT)), dim3(W * 32), smem, st, x, w, p, RowsNorm(), RowsKv()));
  return 0;
}
template <int NT, int S>
static int launch_norm_rows(const bf16* w, const GemmParams& p, const RowsNorm& nm, const RowsKv& kv, cudaStream_t st) {
  auto kern = gemm_rows_kernel<8, NT, 1, false, S, true>;
  const int smem = rows_smem(8, NT, 0, S) + p.T * norm_row_bytes(p.K);
  // the function's limit, for every size: one set for this call could be lowered by another thread's before the launch
  KGE_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_smem(8, NT, 0, S) + 8 * norm_row_bytes(32 * 8 * kNormVecs)));
  KGE_CUDA_OK(launch_pdl(kern, dim3((p.N + 8 * NT - 1) / (8 * NT)), dim3(8 * 32), smem, st, nullptr, w, p, nm, kv));
  return 0;
}
template <bool GATED>
static int launch_rows(const bf16* x, const bf16* w, const GemmParams& p, cudaStream_t st) {
  if constexpr (GATED) {
    return p.T <= 8 ? launch_rows_as<8, 1, 1, true, 3>(x, w, p, st) : launch_rows_as<8, 1, 2, true, 3>(x, w, p, st);
  } else {
    if (p.N <= 8 * 148 && p.K >= 2048) return p.T <= 8 ? launch_rows_as<16, 1, 1, false, 4>(x, w, p, st) : launch_rows_as<16, 1, 2, false, 3>(x, w, p, st);
    if (p.N < 16 * 148) return p.T <= 8 ? launch_rows_as<8, 1, 1, false, 4>(x, w, p, st) : launch_rows_as<8, 1, 2, false, 3>(x, w, p, st);
    return p.T <= 8 ? launch_rows_as<8, 2, 1, false, 3>(x, w, p, st) : launch_rows_as<8, 2, 2, false, 3>(x, w, p, st);
  }
}

// Whether `rows` weight rows (gated: gate and up rows together) of K numbers for T tokens go to the kernel above: up to 8
// tokens it wins up to where the vocabulary projections begin, whose many small tiles suit the persistent TMA kernel (50272 x 768:
// 13.7 us there, 20 here; 128256 x 2048: 77 and 88); with both token halves in use every weight byte drags a token byte along, so
// only matrices up to 16M weights (4096 x 4096, 16 tokens: 9.0 against 9.3; 2048 x 8192: 12.5 against 10.2, 28672 x 4096: 47.1
// against 45.7).  (16 warps per CTA where 8-row tiles leave SMs without work and K is long: 768 x 3072, 3.9 -> 2.2 us.)
static bool use_rows(int T, int rows, int K) {
  if (!tunable(TUN_GEMM_WIDE) || rows > 32768) return false;
  return T <= 8 || (T <= kRowsMaxT && (int64_t)rows * K <= (int64_t)1 << 24 && K <= 4096);
}
