// Causal grouped-query attention over the paged cache, one warp per (token,
// query head), 32-bit arithmetic throughout: the attention of the 32-bit path
// and the check beside the tensor-core kernel.
//
// garuda/src/llama/mod.rs:793-818: query head h reads kv head h / g; score
// s_j = dot(q, K_j) * scale with the scale multiplied after the dot; keys j in
// [start, pos], start = max(0, pos + 1 - window) (garuda/src/cache/mod.rs:333-338);
// softmax with the maximum subtracted (garuda/src/simd/mod.rs:132-158); then the
// sum of p_j V_j in key order, 32 keys by themselves and the 32s added up. Keys are walked 32 at a time from `start`, with
// a running maximum and sum, so the result for a token does not depend on what
// else is in the batch or on how its prompt was cut.
//
// Options that other designs use, each off at its neutral value: `softcap` c > 0 replaces a score
// by c tanh(s / c) (after the scale); `keep_first` n > 0 lets a windowed query also read the first
// n positions of its request (at their true positions); `sink` adds one to the softmax's
// denominator, an entry of score zero that carries no value: p_j = exp(s_j) / (1 + sum exp(s_k));
// `sink_v` (one learned number per query head) adds exp(sink_v[h]) there instead, unscaled; `r1`, `r2`
// (per query head) take r1 ln(1 + r2 (i - j)) off the score of key j for the query at i; `chunk` n > 0
// lets a query read only the keys of its own stretch of n positions, floor(j / n) = floor(i / n),
// counted from the request's first position.
#include "common.cuh"

namespace {

constexpr int WARPS = 4;

// MAX_HD: the widest head this instance takes. A value row is `v_hd` wide in its pool, of which the
// first `vd` channels are summed (vd = v_hd = hd for ordinary attention; a mixer whose keys and
// values are parts of one cached vector passes the same pool twice and a narrower vd).
template <typename T, int MAX_HD>
__global__ void __launch_bounds__(WARPS * 32)
attention_simple_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                        const int32_t* __restrict__ block_table, int table_width,
                        const int32_t* __restrict__ cu_q, const int32_t* __restrict__ kv_lens,
                        const int32_t* __restrict__ token_req, T* __restrict__ out, int Hq, int Hkv, int hd,
                        int v_hd, int vd, float scale, int window, int page_size, float softcap, int keep_first,
                        int sink, const float* __restrict__ sink_v, const float* __restrict__ r1,
                        const float* __restrict__ r2, int chunk) {
  __shared__ float q_s[WARPS][MAX_HD];
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.y * WARPS + warp;
  if (h >= Hq) return;
  const int r = token_req[t];
  const int q_len = cu_q[r + 1] - cu_q[r];
  const int pos = kv_lens[r] - q_len + (t - cu_q[r]);
  const int start = chunk > 0 ? (pos / chunk) * chunk : window > 0 ? max(0, pos + 1 - window) : 0;
  const float far1 = r1 ? r1[h] : 0.f, far2 = r2 ? r2[h] : 0.f;
  const int kvh = h / (Hq / Hkv);
  const int32_t* table = block_table + (size_t)r * table_width;

  const T* qr = q + ((size_t)t * Hq + h) * hd;
  for (int c = lane; c < hd; c += 32) q_s[warp][c] = gb::to_float<T>(qr[c]);
  __syncwarp();

  const int nacc = (vd + 31) / 32;
  float acc[MAX_HD / 32];
#pragma unroll
  for (int i = 0; i < MAX_HD / 32; ++i) acc[i] = 0.f;
  float m = -INFINITY, l = 0.f;

  // two stretches of keys: the kept first positions below the window, then the window
  const int kept = start > 0 ? min(keep_first, start) : 0;
  const int n_blocks_kept = (kept + 31) / 32;
  const int n_blocks = n_blocks_kept + (pos - start + 32) / 32;
  for (int blk = 0; blk < n_blocks; ++blk) {
    const bool in_kept = blk < n_blocks_kept;
    const int base = in_kept ? blk * 32 : start + (blk - n_blocks_kept) * 32;
    const int last = in_kept ? kept - 1 : pos;
    const int j = base + lane;
    const bool valid = j <= last;
    long long row = -1;  // row of this lane's key in the pool, in units of hd elements
    if (valid) {
      const int page = table[j / page_size];
      if (page >= 0) row = ((long long)page * Hkv + kvh) * page_size + (j % page_size);
    }
    float s = -INFINITY;
    if (row >= 0) {
      const T* kr = k_pool + row * hd;
      // eight interleaved sums, added up as a tree: less rounding than one sum of hd terms
      float d8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      int c = 0;
      for (; c + 8 <= hd; c += 8)
#pragma unroll
        for (int e = 0; e < 8; ++e) d8[e] = fmaf(q_s[warp][c + e], gb::to_float<T>(kr[c + e]), d8[e]);
      for (int e = 0; c + e < hd; ++e) d8[0] = fmaf(q_s[warp][c + e], gb::to_float<T>(kr[c + e]), d8[0]);
      s = (((d8[0] + d8[1]) + (d8[2] + d8[3])) + ((d8[4] + d8[5]) + (d8[6] + d8[7]))) * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      if (r1) s -= far1 * log1pf(far2 * (float)(pos - j));
    }
    const float m_new = fmaxf(m, gb::warp_max(s));
    if (m_new == -INFINITY) continue;          // a block without a single stored key
    const float p = row >= 0 ? expf(s - m_new) : 0.f;
    const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
    l = l * corr + gb::warp_sum(p);
    m = m_new;
    float part[MAX_HD / 32];       // the block's keys summed by themselves, then added to the keys in front
#pragma unroll
    for (int i = 0; i < MAX_HD / 32; ++i) part[i] = 0.f;
    const int n_here = min(32, last - base + 1);
    for (int jj = 0; jj < n_here; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const long long rj = __shfl_sync(0xffffffffu, row, jj);
      if (rj < 0) continue;
      const T* vr = v_pool + rj * v_hd;
#pragma unroll
      for (int i = 0; i < MAX_HD / 32; ++i) {
        const int c = lane + 32 * i;
        if (i < nacc && c < vd) part[i] = fmaf(pj, gb::to_float<T>(vr[c]), part[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < MAX_HD / 32; ++i) acc[i] = fmaf(acc[i], corr, part[i]);
  }
  if (sink_v && m != -INFINITY) l += expf(sink_v[h] - m);
  else if (sink && m != -INFINITY) l += expf(-m);
  const float inv = l > 0.f ? 1.0f / l : 0.f;
  T* o = out + ((size_t)t * Hq + h) * vd;
#pragma unroll
  for (int i = 0; i < MAX_HD / 32; ++i) {
    const int c = lane + 32 * i;
    if (i < nacc && c < vd) o[c] = gb::from_float<T>(acc[i] * inv);
  }
}

// ---- 32-bit prompts: the same arithmetic in tiles ------------------------------------------------
//
// A warp per (token, head) reads every key for itself (500 tokens of 32 heads of 64: 0.9 ms). Here a CTA takes 64 consecutive
// (token, head of a kv head's group) rows of a request against 32 keys at a time in shared memory, every number by
// the same operations in the same order as above: the eight interleaved sums of a score and their tree, a block's maximum, its
// exponentials' sum as the warp's tree, a block's values by themselves in the order of the keys. So a token's bits do not depend on
// which of the two kernels ran. Plain attention without a window; heads of 64 or 128 channels.
// What bounds it: shared memory (a thread's 4 x 2 scores read 6 numbers for 8 multiply-adds) and, with few
// long rows, the chain of a block's barriers: prompts of 125 and 375 tokens, 32 heads over 4, take 95 us (a warp per row: 0.9 ms).
constexpr int TR = 64, TK = 32;              // rows and keys of a tile
constexpr int T32 = 256;                     // threads

// two 32-bit multiply-adds in one instruction, on numbers that lie side by side
using pair_t = unsigned long long;
struct __align__(16) pair2_t { pair_t a, b; };
__device__ __forceinline__ void fma2(pair_t& d, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ pair_t make_pair(float lo, float hi) {
  pair_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 both(pair_t p) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(p));
  return f;
}

template <int HD>
struct TileSmem {
  float q[TR][HD + 4], k[2][TK][HD + 4], v[2][TK][HD + 4], p[TR][TK + 4], corr[TR];
  int limit[TR];                             // the last key that a row reads
};

__device__ __forceinline__ void copy_16(float* smem, const float* gmem, bool valid) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}

// grid (tiles of the longest request's rows, Hkv, R)
template <int HD>
__global__ void __launch_bounds__(T32, 2)
attention_tile32_kernel(const float* __restrict__ q, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                        const int32_t* __restrict__ block_table, int table_width, const int32_t* __restrict__ cu_q,
                        const int32_t* __restrict__ kv_lens, float* __restrict__ out, int Hq, int Hkv, float scale, int page_size) {
  constexpr int WARPS_T = T32 / 32, RPW = TR / WARPS_T;          // rows of a warp in the softmax
  constexpr int RV = TR * HD / 4 / T32;                          // rows of a thread's values (by four channels)
  extern __shared__ __align__(16) unsigned char raw[];
  TileSmem<HD>& sm = *reinterpret_cast<TileSmem<HD>*>(raw);
  const int r = blockIdx.z, kvh = blockIdx.y, G = Hq / Hkv;
  // (the last rows, which read the most keys, first)
  const int t0 = cu_q[r], n = cu_q[r + 1] - t0, row0 = (gridDim.x - 1 - blockIdx.x) * TR, rows = min(TR, n * G - row0);
  if (rows <= 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pos0 = kv_lens[r] - n;                               // the position of the request's first token of the step
  const int last = pos0 + (row0 + rows - 1) / G;                 // the last key that a row of the tile reads
  const int blocks = last / TK + 1;
  const int32_t* table = block_table + (size_t)r * table_width;
  auto where = [&](int row) {                                    // (token, head) row of q and out
    const int i = row0 + row;
    return (size_t)(t0 + i / G) * Hq + kvh * G + i % G;
  };
  auto load = [&](int b) {
    for (int i = tid; i < TK * (HD / 4); i += T32) {
      const int key = i / (HD / 4), c = i % (HD / 4) * 4, j = b * TK + key;
      const int page = j <= last ? table[j / page_size] : -1;
      const size_t at = page >= 0 ? (((size_t)page * Hkv + kvh) * page_size + j % page_size) * HD + c : 0;
      copy_16(&sm.k[b & 1][key][c], k_pool + at, page >= 0);
      copy_16(&sm.v[b & 1][key][c], v_pool + at, page >= 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0);
  for (int row = warp; row < TR; row += WARPS_T) {
    const float* from = q + (row < rows ? where(row) * HD : 0);
    for (int c = lane; c < HD; c += 32) sm.q[row][c] = row < rows ? from[c] : 0.f;
    if (lane == 0) sm.limit[row] = row < rows ? pos0 + (row0 + row) / G : -1;
  }
  // the softmax: a warp has RPW rows, a lane a key
  float m[RPW], l[RPW];
#pragma unroll
  for (int i = 0; i < RPW; ++i) m[i] = -INFINITY, l[i] = 0.f;
  // the values: a thread has RV rows and four channels
  const int c4 = tid % (HD / 4) * 4, rv = tid / (HD / 4) * RV;
  pair_t acc[RV][2];
#pragma unroll
  for (int i = 0; i < RV; ++i) acc[i][0] = acc[i][1] = 0ull;
  // the scores: four rows (four apart), two keys (eight apart)
  const int rs = (warp & 3) * 16 + (lane >> 3), ks = (warp >> 2) * 16 + (lane & 7);
  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                       // the block has landed; everyone is done with the one in front
    if (b + 1 < blocks) load(b + 1);
    {
      pair_t d8[4][2][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) d8[i][j][e] = 0ull;
#pragma unroll 4
      for (int c = 0; c < HD; c += 8) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          pair2_t x[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const pair2_t*>(&sm.q[rs + 4 * i][c + 4 * half]);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const pair2_t y = *reinterpret_cast<const pair2_t*>(&sm.k[b & 1][ks + 8 * j][c + 4 * half]);
#pragma unroll
            for (int i = 0; i < 4; ++i) fma2(d8[i][j][2 * half], x[i].a, y.a), fma2(d8[i][j][2 * half + 1], x[i].b, y.b);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 d01 = both(d8[i][j][0]), d23 = both(d8[i][j][1]), d45 = both(d8[i][j][2]), d67 = both(d8[i][j][3]);
          sm.p[rs + 4 * i][ks + 8 * j] = (((d01.x + d01.y) + (d23.x + d23.y)) + ((d45.x + d45.y) + (d67.x + d67.y))) * scale;
        }
    }
    __syncthreads();
    const int key = b * TK + lane;
    const bool stored = key <= last && table[key / page_size] >= 0;
#pragma unroll
    for (int i = 0; i < RPW; ++i) {
      const int row = warp * RPW + i;
      const bool seen = stored && key <= sm.limit[row];
      const float s = seen ? sm.p[row][lane] : -INFINITY;
      const float m_new = fmaxf(m[i], gb::warp_max(s));
      float p = 0.f, corr = 1.f;           // (a block without a stored key that the row reads changes nothing)
      if (m_new != -INFINITY) {
        p = seen ? expf(s - m_new) : 0.f;
        corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
        l[i] = l[i] * corr + gb::warp_sum(p);
        m[i] = m_new;
      }
      sm.p[row][lane] = p;
      if (lane == 0) sm.corr[row] = corr;
    }
    __syncthreads();
    pair_t part[RV][2];
#pragma unroll
    for (int i = 0; i < RV; ++i) part[i][0] = part[i][1] = 0ull;
    // A row must not meet the values of keys behind its own, which may be anything: where the block holds such keys for some row
    // the sums look at each. (A zero weight adds an exact zero otherwise.)
    if (b * TK + TK - 1 <= pos0 + row0 / G) {
#pragma unroll
      for (int j = 0; j < TK; j += 4) {
        pair2_t y[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = *reinterpret_cast<const pair2_t*>(&sm.v[b & 1][j + e][c4]);
#pragma unroll
        for (int i = 0; i < RV; ++i) {
          const float4 p4 = *reinterpret_cast<const float4*>(&sm.p[rv + i][j]);
          const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const pair_t pp = make_pair(p[e], p[e]);
            fma2(part[i][0], pp, y[e].a), fma2(part[i][1], pp, y[e].b);
          }
        }
      }
    } else {
      int seen[RV];                        // how many of the block's keys a row reads
#pragma unroll
      for (int i = 0; i < RV; ++i) seen[i] = sm.limit[rv + i] - b * TK + 1;
#pragma unroll 4
      for (int j = 0; j < TK; ++j) {
        const pair2_t y = *reinterpret_cast<const pair2_t*>(&sm.v[b & 1][j][c4]);
#pragma unroll
        for (int i = 0; i < RV; ++i) {
          const float p = sm.p[rv + i][j];
          const pair_t pp = make_pair(p, p);
          if (j < seen[i]) fma2(part[i][0], pp, y.a), fma2(part[i][1], pp, y.b);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < RV; ++i) {
      const float corr = sm.corr[rv + i];
      const pair_t cc = make_pair(corr, corr);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        fma2(part[i][e], acc[i][e], cc);
        acc[i][e] = part[i][e];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RPW; ++i)
    if (lane == 0) sm.corr[warp * RPW + i] = l[i] > 0.f ? 1.0f / l[i] : 0.f;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RV; ++i) {
    if (rv + i >= rows) continue;
    const float inv = sm.corr[rv + i];
    const float2 lo = both(acc[i][0]), hi = both(acc[i][1]);
    *reinterpret_cast<float4*>(out + where(rv + i) * HD + c4) = make_float4(lo.x * inv, lo.y * inv, hi.x * inv, hi.y * inv);
  }
}

template <int HD>
int launch_tile32(const float* q, const float* k_pool, const float* v_pool, const int32_t* block_table, int table_width,
                  const int32_t* cu_q, const int32_t* kv_lens, float* out, int R, int max_q, int Hq, int Hkv, float scale, int page_size,
                  cudaStream_t stream) {
  static gb::OncePerDevice configured;
  if (configured.needed()) {
    const cudaError_t e = cudaFuncSetAttribute(attention_tile32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem<HD>));
    if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "attention_tile32: %s", cudaGetErrorString(e));
    configured.done();
  }
  const long long tiles = ((long long)max_q * (Hq / Hkv) + TR - 1) / TR;
  attention_tile32_kernel<HD><<<dim3((unsigned)tiles, Hkv, R), T32, sizeof(TileSmem<HD>), stream>>>(
      q, k_pool, v_pool, block_table, table_width, cu_q, kv_lens, out, Hq, Hkv, scale, page_size);
  return gb::check_launch("attention_tile32");
}

}  // namespace

// Plain causal attention of a 32-bit prompt, bit for bit what gb_attention_simple gives. hd 64 or 128; q, out and the pools start on 16
// bytes; max_q: the most tokens that a request of the step has.
GB_EXPORT int gb_attention_tile32(const float* q, const float* k_pool, const float* v_pool, const int32_t* block_table, int table_width,
                                  const int32_t* cu_q, const int32_t* kv_lens, float* out, int R, int max_q, int Hq, int Hkv, int hd,
                                  float scale, int page_size, cudaStream_t stream) {
  if (R <= 0 || max_q <= 0) return GB_OK;
  if (Hkv < 1 || Hq % Hkv || Hkv > 65535 || R > 65535) return gb::fail(GB_BAD_ARGUMENT, "attention_tile32: %d query heads for %d kv heads, %d requests", Hq, Hkv, R);
  if (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out) & 15) return gb::fail(GB_BAD_ARGUMENT, "attention_tile32: 16-byte addresses");
  if (hd == 64) return launch_tile32<64>(q, k_pool, v_pool, block_table, table_width, cu_q, kv_lens, out, R, max_q, Hq, Hkv, scale, page_size, stream);
  if (hd == 128) return launch_tile32<128>(q, k_pool, v_pool, block_table, table_width, cu_q, kv_lens, out, R, max_q, Hq, Hkv, scale, page_size, stream);
  return gb::fail(GB_UNSUPPORTED, "attention_tile32: heads of %d channels", hd);
}

// v_hd: width of a value row in its pool; vd: how many of its first channels are the value
// (out is [T, Hq, vd]). Ordinary attention passes hd for both.
GB_EXPORT int gb_attention_simple(const void* q, const void* k_pool, const void* v_pool, int dtype,
                                  const int32_t* block_table, int table_width, const int32_t* cu_q,
                                  const int32_t* kv_lens, const int32_t* token_req, void* out, int T,
                                  int Hq, int Hkv, int hd, int v_hd, int vd, float scale, int window,
                                  int page_size, float softcap, int keep_first, int sink, const float* sink_v,
                                  const float* r1, const float* r2, int chunk, cudaStream_t stream) {
  if (T <= 0) return GB_OK;
  constexpr int WIDEST = 1024;
  if (hd > WIDEST || hd < 1)
    return gb::fail(GB_UNSUPPORTED, "attention: head_dim %d is outside 1..%d", hd, WIDEST);
  if (vd < 1 || vd > v_hd || vd > WIDEST)
    return gb::fail(GB_BAD_ARGUMENT, "attention: %d value channels of rows %d wide", vd, v_hd);
  if (Hkv < 1 || Hq % Hkv) return gb::fail(GB_BAD_ARGUMENT, "attention: %d query heads for %d kv heads", Hq, Hkv);
  if ((r1 == nullptr) != (r2 == nullptr)) return gb::fail(GB_BAD_ARGUMENT, "attention: the distance term takes both of its numbers");
  if (chunk < 0 || (chunk > 0 && (window > 0 || keep_first > 0)))
    return gb::fail(GB_BAD_ARGUMENT, "attention: a stretch of %d positions goes with no window", chunk);
  dim3 grid(T, (Hq + WARPS - 1) / WARPS);
  return GB_DISPATCH_DTYPE(dtype, TT, [&]() -> int {
    if (hd <= 256 && vd <= 256)
      attention_simple_kernel<TT, 256><<<grid, WARPS * 32, 0, stream>>>(
          (const TT*)q, (const TT*)k_pool, (const TT*)v_pool, block_table, table_width, cu_q, kv_lens,
          token_req, (TT*)out, Hq, Hkv, hd, v_hd, vd, scale, window, page_size, softcap, keep_first, sink, sink_v, r1, r2, chunk);
    else
      attention_simple_kernel<TT, WIDEST><<<grid, WARPS * 32, 0, stream>>>(
          (const TT*)q, (const TT*)k_pool, (const TT*)v_pool, block_table, table_width, cu_q, kv_lens,
          token_req, (TT*)out, Hq, Hkv, hd, v_hd, vd, scale, window, page_size, softcap, keep_first, sink, sink_v, r1, r2, chunk);
    return gb::check_launch("attention_simple");
  });
}
