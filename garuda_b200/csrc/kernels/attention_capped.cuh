// What the kernels of the attention with capped scores, kept first positions, sinks, a distance term or a chunked mask share: the
// argument block, the mask, and the hand-over from the entry point to the tcgen05 kernel for prompt portions.
#pragma once

#include "common.cuh"

namespace capped {

constexpr int ROWS_DECODE = 16;     // a request with at most this many (token, head-of-group) rows is a decode request

struct Params {
  const __nv_bfloat16* q;        // [T, Hq, HD]
  const __nv_bfloat16* k_pool;   // [pages, Hkv, page_size, HD]
  const __nv_bfloat16* v_pool;   // [pages, Hkv, page_size, VD]
  __nv_bfloat16* out;            // [T, Hq * VD]
  const int32_t* block_table;
  const int32_t* cu_q;
  const int32_t* kv_lens;
  float* partials;               // [R, Hkv, splits, ROWS_DECODE, PR] (DECODE with splits > 1)
  int table_width, Hq, Hkv, g, window, keep_first, page_size, sink, splits;
  float scale, softcap;
  const float* sink_v;           // [Hq] or null: a learned sink per query head
  const float* r1;               // [Hq] or null: the distance term's two numbers per query head
  const float* r2;
  int chunk;                     // > 0: a query reads its own stretch of this many positions (no window then)
};

// First position that the query at `pos` reads (kept first positions aside).
__device__ __forceinline__ int first_seen(const Params& p, int pos) {
  if (p.chunk > 0) return pos / p.chunk * p.chunk;
  return p.window > 0 ? max(0, pos + 1 - p.window) : 0;
}

// True if the tcgen05 kernel takes this shape: widths of 64 or 128, a power-of-two group, pages of 8 to 64 keys, a positive scale.
bool tc_takes(const Params& p, long long pages, int R);
// Launches it for every request with more than ROWS_DECODE rows. Returns a GbStatus.
int launch_tc(const Params& p, int T, long long pages, int R, int max_q_len, cudaStream_t stream);
int tc_error_check();
int tc_set_error_sink(int* host_word);

}  // namespace capped
