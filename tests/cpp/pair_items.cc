// The prompt attention kernel's search for its work (csrc/attn_pair.cuh), 32 lanes as threads that meet at every warp operation.
// Input: H KV per by_request B, then query_start_loc; CTAs one after another: "x y z" each until end of file.
// Output, a line per CTA: request, kv head, first token (negative: no work).
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <barrier>
#include <thread>
#include <vector>

using std::max;
using std::min;
static std::barrier<> meet(32);
static uint32_t shared_val[32];
static thread_local int lane;

static uint32_t exchange(uint32_t v, int from) {
  shared_val[lane] = v;
  meet.arrive_and_wait();
  const uint32_t r = shared_val[from];
  meet.arrive_and_wait();
  return r;
}
static int __shfl_up_sync(uint32_t, int v, int o) { return (int)exchange((uint32_t)v, lane >= o ? lane - o : lane); }
static int __shfl_sync(uint32_t, int v, int l) { return (int)exchange((uint32_t)v, l & 31); }
static uint32_t __ballot_sync(uint32_t, bool p) {
  shared_val[lane] = p;
  meet.arrive_and_wait();
  uint32_t r = 0;
  for (int i = 0; i < 32; ++i) r |= (shared_val[i] & 1u) << i;
  meet.arrive_and_wait();
  return r;
}
static int __ffs(uint32_t v) { return __builtin_ffs((int)v); }

struct Found { int b, kvh, tok0; };

static Found find(int bx, int by, int bz, int flat, int KV, int TI, const int32_t* qsl, const int32_t* seq_lens, const int32_t* block_table) {
  const int box_rows = 64, bs_shift = 6, max_blocks = 1;
#include KERNEL_PART
  (void)id0; (void)seq_len;
  return {b, kvh, tok0};
}

int main() {
  int H, KV, per, by_request, B;
  if (scanf("%d %d %d %d %d", &H, &KV, &per, &by_request, &B) != 5) return 1;
  std::vector<int32_t> qsl(B + 1), lens(B), table(B);
  for (auto& q : qsl)
    if (scanf("%d", &q) != 1) return 1;
  for (int b = 0; b < B; ++b) lens[b] = qsl[b + 1] - qsl[b];
  std::vector<int> cta;
  for (int v; scanf("%d", &v) == 1;) cta.push_back(v);
  std::vector<Found> out(cta.size() / 3);
  std::vector<std::thread> lanes;
  for (int l = 0; l < 32; ++l)
    lanes.emplace_back([&, l] {
      lane = l;
      for (size_t i = 0; i < out.size(); ++i) {
        const Found f = find(cta[3 * i], cta[3 * i + 1], cta[3 * i + 2], by_request ? B : 0, KV, per * (128 / (H / KV)), qsl.data(), lens.data(), table.data());
        if (l == 0) out[i] = f;
      }
    });
  for (auto& t : lanes) t.join();
  for (auto& f : out) printf("%d %d %d\n", f.b, f.kvh, f.tok0);
  return 0;
}
