// A few rows normalised and projected in one launch (gemm_rows.cuh): what the engine's small steps of OPT models use in the place of a
// norm kernel, a projection and the write of keys and values into the cache (which needs no rotation there).
#pragma once
#include <stdint.h>

namespace kge {
struct RowsNorm {                                   // LayerNorm of the rounded sum of the residual stream and add
  const void *res = nullptr, *add = nullptr;        // [T, K]; add may be null
  void* res_out = nullptr;                          // [T, K]: the sum (with add only; another buffer than res)
  const void *w = nullptr, *b = nullptr;
  float eps = 0.f;
};
struct RowsKv {                                     // columns from q_cols on are keys, then values: [KV, hd] each
  void *kc = nullptr, *vc = nullptr;                // [blocks, KV, bs, hd]; null: no such columns
  const int64_t* slots = nullptr;
  int q_cols = 0, KV = 0, hd = 0, bs = 0;
};
}  // namespace kge

// norm_gemm_ok: whether these sizes are taken
extern "C" bool kge_norm_gemm_ok(int T, int N, int K);
extern "C" int kge_norm_gemm(void* y, const kge::RowsNorm& nm, const void* w, const void* bias, int T, int N, int K, int act, const kge::RowsKv& kv, void* stream);
extern "C" int kge_norm_gemm_f16(void* y, const kge::RowsNorm& nm, const void* w, const void* bias, int T, int N, int K, int act, const kge::RowsKv& kv, void* stream);
