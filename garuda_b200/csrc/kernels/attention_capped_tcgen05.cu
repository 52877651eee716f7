// Prompt portions of the attention of attention_capped_mma.cu (capped scores, a window that keeps a request's first positions, a
// sink, a distance term, a chunked mask) on the fifth-generation tensor cores, for keys and values of 64 or 128 channels.
//
// A CTA takes 128 query rows, (token, head-of-group) pairs of one kv head of one request, and walks their keys 64 at a time: first
// the tiles that hold kept first positions below the window, then the window's. Two CTAs share an SM, so that one computes exponentials
// while the other waits for tensor memory.
//   warp 0     TMA: the query tile (3-D boxes [tokens][group][64]), then keys and values, one 4-D box per page and block of 64 channels.
//              Pages that are not there or that no row reads are asked for beyond the pool's end, which fills their rows with zeros.
//   warp 1     one elected lane: S = Q K^T a tile ahead into one of two S buffers in tensor memory, O += P V of the tile whose softmax just ended.
//   warps 2-5  a thread owns a query row: its 64 scores, the cap, the distance term, the mask on tiles that some row does not see whole,
//              exp2 against the running maximum (where it grows for some row of a warp, that warp rescales O, which stays in tensor
//              memory: a reference that lags behind would round the largest weights, as latent_attention_tcgen05.cu tells), P in
//              bfloat16 over the scores read. The sink joins the denominator at the end.
// What bounds it: instruction issue of the softmax warps. The cap's polynomial is nine operations a score, taken two scores an
// instruction (f32x2); a score's exponential and sum are four more. A prompt of 2,048 tokens, 32 heads over 4 of 64, window 1,024, cap 30 and
// sink: 126 us with mma.sync, 79 here, behind a flushed L2 (72 in a row, since products are issued by an elected lane; a branch a pair of scores for those beyond the cap, which the fetch of instructions waited for, cost 17
// more).
// Every wait is bounded; a wait that runs out sets the error word and the CTA winds down.
#include "attention_capped.cuh"
#include "error_word.cuh"
#include "tc_common.cuh"
#include "tc_host.cuh"

#ifndef GB_KEY_DIM
#define GB_KEY_DIM 64
#endif
#ifndef GB_VALUE_DIM
#define GB_VALUE_DIM 64
#endif

#if (GB_KEY_DIM == 64 || GB_KEY_DIM == 128) && (GB_VALUE_DIM == 64 || GB_VALUE_DIM == 128)

namespace {

using namespace tc;
using capped::first_seen;
using capped::Params;

constexpr int HD = GB_KEY_DIM, VD = GB_VALUE_DIM;
constexpr int KBLOCKS = HD / 64, VBLOCKS = VD / 64;             // blocks of 64 channels: one swizzled 128-byte row each
constexpr int QROWS = 128, KT = 64;
constexpr int ROW_BYTES = 128;
constexpr int Q_BLOCK = QROWS * ROW_BYTES, K_BLOCK = KT * ROW_BYTES;
constexpr int Q_BYTES = KBLOCKS * Q_BLOCK, K_BYTES = KBLOCKS * K_BLOCK, V_BYTES = VBLOCKS * K_BLOCK;
constexpr int STAGE_BYTES = K_BYTES + V_BYTES;
// two CTAs an SM, and not three (each takes half of the tensor memory): 80 to 96 KB each
constexpr int STAGES = (98304 - Q_BYTES) / STAGE_BYTES > 4 ? 4 : (98304 - Q_BYTES) / STAGE_BYTES;
constexpr int TILE_BYTES = Q_BYTES + STAGES * STAGE_BYTES;
static_assert(STAGES >= 2 && TILE_BYTES >= 77824, "two CTAs an SM");
constexpr int S_BUFS = 2, O_COL0 = S_BUFS * KT, TMEM_COLS = 256;
static_assert(O_COL0 + VD <= TMEM_COLS, "tensor memory layout");
constexpr int THREADS = 64 + QROWS;
constexpr float LOG2E = 1.4426950408889634f;

struct Misc {
  uint64_t q_full, full[STAGES], empty[STAGES], s_ready[S_BUFS], p_ready[S_BUFS], o_ready;
  uint32_t tmem_base;
  int abort;
};
constexpr int SMEM_BYTES = TILE_BYTES + (int)sizeof(Misc);

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void st_shared_zero(uint32_t addr) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0u) : "memory");
}
// two 32-bit operations in one instruction
using pair_t = unsigned long long;
__device__ __forceinline__ pair_t make_pair(float lo, float hi) {
  pair_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack(pair_t p, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p)); }
__device__ __forceinline__ pair_t mul2(pair_t a, pair_t b) {
  pair_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
  pair_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// tanh beyond [-1, 1] by way of the exponential, as in attention_capped_mma.cu
__device__ __forceinline__ float tanh_exp2(float x) {
  x = fminf(fmaxf(x, -15.f), 15.f);
  const float t = fast_exp2(x * (2.0f * LOG2E));
  return 1.0f - __fdividef(2.0f, t + 1.0f);
}

// grid (query tiles of the longest request, Hkv, R)
template <bool CAP, bool FAR>
__global__ void __launch_bounds__(THREADS, 2)
capped_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                 const Params p, int pages) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Misc& mc = *reinterpret_cast<Misc*>(smem_raw + TILE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t q_s = smem_u32(smem_raw), kv_s = q_s + Q_BYTES;   // stage s: keys at kv_s + s * STAGE_BYTES, values K_BYTES behind
  if ((q_s & 1023u) != 0) {                                        // the swizzle needs it; never seen
    if (threadIdx.x == 0) gb_err::report(ERR_WAIT_DRAIN);
    return;
  }
  const int r = blockIdx.z, kvh = blockIdx.y;
  // The batch's lengths and tables were copied in before the step's first kernel.
  const int q_begin = p.cu_q[r], q_len = p.cu_q[r + 1] - q_begin;
  const int tokens_per_tile = QROWS / p.g;
  const int tok0 = (int)(gridDim.x - 1 - blockIdx.x) * tokens_per_tile;      // the last rows, which may read the most keys, first
  if (q_len * p.g <= capped::ROWS_DECODE || tok0 >= q_len) return;           // a decode request, or past its end
  const int ntok = min(tokens_per_tile, q_len - tok0), rows = ntok * p.g;
  const int pos0 = p.kv_lens[r] - q_len + tok0;
  const int lo = first_seen(p, pos0), hi = pos0 + ntok - 1;        // the first and last key that a row reads (kept ones aside)
  const int last_start = first_seen(p, hi);
  const int tile_begin = lo / KT;
  const int kept_tiles = p.keep_first > 0 ? min((p.keep_first + KT - 1) / KT, tile_begin) : 0;
  const int n_tiles = kept_tiles + hi / KT + 1 - tile_begin;
  auto first_key = [&](int t) { return (t < kept_tiles ? t : tile_begin + t - kept_tiles) * KT; };
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&mc.q_full), 1);
    mbar_init(smem_u32(&mc.o_ready), 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&mc.full[s]), 1);
      mbar_init(smem_u32(&mc.empty[s]), 1);
    }
    for (int b = 0; b < S_BUFS; ++b) {
      mbar_init(smem_u32(&mc.s_ready[b]), 1);
      mbar_init(smem_u32(&mc.p_ready[b]), QROWS);
    }
    mc.abort = 0;
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tensormap(&q_map);
    prefetch_tensormap(&k_map);
    prefetch_tensormap(&v_map);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&mc.tmem_base), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = mc.tmem_base;
  volatile int* abort_s = &mc.abort;
  gb::pdl_launch_dependents();
  gb::pdl_wait();      // queries and this step's keys and values come from the kernel in front

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    const int per_tile = KT / p.page_size;                         // 1 to 8 pages, a lane each
    const int32_t* table = p.block_table + (size_t)r * p.table_width;
    int loaded = 0;                                                // tiles asked for
    if (lane == 0) {
      mbar_arrive_expect_tx(smem_u32(&mc.q_full), Q_BYTES);
#pragma unroll
      for (int b = 0; b < KBLOCKS; ++b) tma_load_3d(q_s + b * Q_BLOCK, &q_map, smem_u32(&mc.q_full), b * 64, kvh * p.g, q_begin + tok0);
    }
    for (int t = 0; t < n_tiles; ++t) {
      const int st = t % STAGES;
      const int first = first_key(t) + lane * p.page_size;
      const bool read = lane < per_tile && first <= hi && (first + p.page_size > lo || first < p.keep_first);
      int page = read ? table[first / p.page_size] : -1;
      if (page < 0 || page >= pages) page = pages;                 // beyond the pool: zeros
      if (lane == 0) {
        if (t >= STAGES && !mbar_wait(smem_u32(&mc.empty[st]), (t / STAGES - 1) & 1)) {
          gb_err::report(ERR_WAIT_EMPTY);
          *abort_s = 1;
        }
        if (!*abort_s) mbar_arrive_expect_tx(smem_u32(&mc.full[st]), STAGE_BYTES);
      }
      __syncwarp();
      if (*abort_s) break;
      if (lane < per_tile) {
        const uint32_t to = kv_s + st * STAGE_BYTES + lane * p.page_size * ROW_BYTES;
#pragma unroll
        for (int b = 0; b < KBLOCKS; ++b) tma_load_4d(to + b * K_BLOCK, &k_map, smem_u32(&mc.full[st]), b * 64, 0, kvh, page);
#pragma unroll
        for (int b = 0; b < VBLOCKS; ++b) tma_load_4d(to + K_BYTES + b * K_BLOCK, &v_map, smem_u32(&mc.full[st]), b * 64, 0, kvh, page);
      }
      loaded = t + 1;
    }
    // the copies in flight land before the CTA's shared memory is given up
    if (lane == 0) {
      bool ok = mbar_wait(smem_u32(&mc.q_full), 0);
      for (int t = loaded > STAGES ? loaded - STAGES : 0; t < loaded; ++t) ok = mbar_wait(smem_u32(&mc.full[t % STAGES]), (t / STAGES) & 1) && ok;
      if (!ok) gb_err::report(ERR_WAIT_DRAIN);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issuer
    const bool leader = elect_one();
    constexpr uint32_t idesc_s = instr_desc_bf16(QROWS, KT);
    constexpr uint32_t idesc_o = instr_desc_bf16(QROWS, VD) | INSTR_B_MN_MAJOR;
    const uint64_t dq0 = smem_desc_sw128(q_s), dk0 = smem_desc_sw128(kv_s), dv0 = smem_desc_sw128_mn(kv_s + K_BYTES, K_BLOCK);
    bool ok = mbar_wait(smem_u32(&mc.q_full), 0);
    if (!ok && lane == 0) gb_err::report(ERR_WAIT_FULL);
    auto issue_s = [&](int t) {
      const int st = t % STAGES, buf = t % S_BUFS;
      if (!mbar_wait(smem_u32(&mc.full[st]), (t / STAGES) & 1)) {
        if (lane == 0) gb_err::report(ERR_WAIT_FULL);
        ok = false;
        return;
      }
      tc_fence_after_sync();
      if (leader) {
#pragma unroll
        for (int b = 0; b < KBLOCKS; ++b)
          mma_bf16_x4(tmem_base + buf * KT, dq0 + (uint64_t)(b * (Q_BLOCK >> 4)), dk0 + (uint64_t)(st * (STAGE_BYTES >> 4) + b * (K_BLOCK >> 4)),
                      idesc_s, 2, 2, b > 0);
        mma_commit(smem_u32(&mc.s_ready[buf]));
      }
      __syncwarp();
    };
    if (ok) issue_s(0);
    for (int t = 0; t < n_tiles && ok; ++t) {
      const int st = t % STAGES, buf = t % S_BUFS;
      if (*abort_s) break;
      // the next tile's scores first: their buffer's probabilities are read by the products issued a turn ago, which end before
      if (t + 1 < n_tiles) issue_s(t + 1);
      if (!ok) break;
      if (!mbar_wait(smem_u32(&mc.p_ready[buf]), (t / S_BUFS) & 1)) {
        if (lane == 0) gb_err::report(ERR_WAIT_ACCUM);
        ok = false;
        break;
      }
      tc_fence_after_sync();
      if (leader) {
        mma_bf16_ts<KT / 16>(tmem_base + O_COL0, tmem_base + buf * KT, dv0 + (uint64_t)(st * (STAGE_BYTES >> 4)), idesc_o, 16 * ROW_BYTES >> 4, t > 0);
        mma_commit(smem_u32(&mc.empty[st]));
        mma_commit(smem_u32(&mc.o_ready));
      }
      __syncwarp();
    }
    if (!ok) *abort_s = 1;
  } else {
    // -------------------------------------------------------------------- softmax warps
    const int quarter = warp & 3;                                  // the TMEM lanes this warp may read
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int row_pos = row < rows ? pos0 + row / p.g : -1;        // no key is valid for a padding row
    const int row_start = row < rows ? first_seen(p, row_pos) : 0;
    const int head = kvh * p.g + row % p.g;
    // A score's unit is what `unit` powers of two the softmax counts for one of it: the raw dot product, or the tanh of its cap
    const float unit = CAP ? p.softcap * LOG2E : p.scale * LOG2E;
    const float pre = CAP ? p.scale / p.softcap : 1.f;
    const float far1 = FAR ? p.r1[head] / unit : 0.f, far2 = FAR ? p.r2[head] : 0.f;      // r1 ln x = r1 log2 x / log2 e
    float m = -INFINITY, l = 0.f;                                  // m: the largest score so far, in units
    bool ok = true;
    auto wait_o = [&](int t) {                                     // until the P V product of tile t has ended
      if (!mbar_wait(smem_u32(&mc.o_ready), t & 1)) {
        if (lane == 0) gb_err::report(ERR_WAIT_ACCUM);
        ok = false;
        *abort_s = 1;
      }
      tc_fence_after_sync();
    };
    for (int t = 0; t < n_tiles; ++t) {
      if (*abort_s) { ok = false; break; }
      const int st = t % STAGES, buf = t % S_BUFS;
      if (!mbar_wait(smem_u32(&mc.s_ready[buf]), (t / S_BUFS) & 1)) {
        if (lane == 0) gb_err::report(ERR_WAIT_ACCUM);
        ok = false;
        *abort_s = 1;
        break;
      }
      tc_fence_after_sync();
      const uint32_t s_addr = lane_addr + buf * KT;
      uint32_t sv[KT / 32][32];
#pragma unroll
      for (int h = 0; h < KT / 32; ++h) tmem_ld_32(s_addr + h * 32, sv[h]);
      const int key0 = first_key(t);
      if (key0 + KT - 1 > hi || key0 < lo) {
        // Value rows that no row reads hold whatever is there (the unwritten end of a page, positions that have left the window): their
        // probabilities are zero, but zero times a stray NaN is not.
        const int key = key0 + row;
        if (row < KT && (key > hi || (key < lo && key >= p.keep_first))) {
#pragma unroll
          for (int b = 0; b < VBLOCKS; ++b)
#pragma unroll
            for (int c = 0; c < ROW_BYTES / 16; ++c) st_shared_zero(kv_s + st * STAGE_BYTES + K_BYTES + b * K_BLOCK + row * ROW_BYTES + c * 16);
        }
        fence_proxy_async();
      }
      tmem_ld_wait();
      auto sc = [&](int c) -> float& { return reinterpret_cast<float&>(sv[c >> 5][c & 31]); };
      if (CAP) {
        // tanh within [-1, 1] as an odd polynomial of degree 13, two scores an instruction; where a score of the warp lies beyond,
        // by way of the exponential for those that do (attention_capped_mma.cu gives the polynomial's error)
        float largest = 0.f;
        const pair_t pre2 = make_pair(pre, pre);
#pragma unroll
        for (int c = 0; c < KT; c += 2) largest = max3(largest, fabsf(sc(c)), fabsf(sc(c + 1)));
        const bool beyond = __any_sync(0xffffffffu, !(largest * pre <= 1.0f));
        if (!beyond) {                                             // the usual case, in one piece: a branch a score is fetched late
          auto k2 = [](float k) { return make_pair(k, k); };
#pragma unroll
          for (int c = 0; c < KT; c += 2) {
            const pair_t x = mul2(make_pair(sc(c), sc(c + 1)), pre2), x2 = mul2(x, x);
            pair_t q = fma2(k2(0.0009637729963287711f), x2, k2(-0.005951283033937216f));
            q = fma2(q, x2, k2(0.019973287358880043f));
            q = fma2(q, x2, k2(-0.05326583608984947f));
            q = fma2(q, x2, k2(0.13319583237171173f));
            q = fma2(q, x2, k2(-0.33332130312919617f));
            q = fma2(q, x2, k2(0.9999997019767761f));
            unpack(mul2(q, x), sc(c), sc(c + 1));
          }
        } else {
#pragma unroll
          for (int c = 0; c < KT; ++c) {
            const float x = sc(c) * pre, x2 = x * x;
            float q = fmaf(0.0009637729963287711f, x2, -0.005951283033937216f);
            q = fmaf(q, x2, 0.019973287358880043f);
            q = fmaf(q, x2, -0.05326583608984947f);
            q = fmaf(q, x2, 0.13319583237171173f);
            q = fmaf(q, x2, -0.33332130312919617f);
            q = fmaf(q, x2, 0.9999997019767761f);
            sc(c) = x2 > 1.0f ? tanh_exp2(x) : q * x;              // (its clamps would turn what is not a number into a score)
          }
        }
      }
      if (FAR) {
#pragma unroll
        for (int c = 0; c < KT; ++c) {
          // a key behind the row (masked below) is given distance zero
          const float dist = (float)max(row_pos - (key0 + c), 0);
          sc(c) = fmaf(-far1, __log2f(fmaf(far2, dist, 1.0f)), sc(c));
        }
      }
      const bool whole = key0 + KT - 1 <= pos0 && (key0 >= last_start || key0 + KT <= p.keep_first);
      if (!whole) {
#pragma unroll
        for (int c = 0; c < KT; ++c) {
          const int j = key0 + c;
          if (!(j <= row_pos && (j >= row_start || j < p.keep_first))) sc(c) = -INFINITY;
        }
      }
      float mx[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < KT; c += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) mx[e] = max3(mx[e], sc(c + e), sc(c + 4 + e));
      const float m_new = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      const bool grown = m != -INFINITY && m_new > m;
      bool waited = false;
      if (t > 0 && __any_sync(0xffffffffu, grown)) {
        wait_o(t - 1);
        waited = true;
        if (!ok) break;
        const float corr = m == -INFINITY ? 1.f : fast_exp2((m - m_new) * unit);
#pragma unroll 1
        for (int h = 0; h < VD / 32; ++h) {
          uint32_t v[32];
          tmem_ld_32(lane_addr + O_COL0 + h * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) * corr);
          tmem_st_32(lane_addr + O_COL0 + h * 32, v);
        }
        l *= corr;
        m = m_new;
      } else if (m == -INFINITY) {
        m = m_new;
      }
      const float neg_m = m == -INFINITY ? 0.f : -m * unit;        // nothing valid yet: avoid inf - inf
#pragma unroll
      for (int c = 0; c < KT; ++c) sc(c) = fast_exp2(fmaf(sc(c), unit, neg_m));
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[KT / 2];
#pragma unroll
      for (int c = 0; c < KT; c += 2) {
        ls[(c >> 1) & 3] += sc(c) + sc(c + 1);
        pk[c >> 1] = pack_bf16(sc(c), sc(c + 1));
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      tmem_st(s_addr, pk);                                         // over the first half of the scores just read
      tmem_st_wait();
      if (t > 0 && !waited) wait_o(t - 1);                         // every phase of the barrier is seen, in order
      tc_fence_before_sync();
      mbar_arrive(smem_u32(&mc.p_ready[buf]));
    }
    if (ok) wait_o(n_tiles - 1);
    if (ok && !*abort_s) {
      if (m != -INFINITY) {
        if (p.sink_v != nullptr) l += fast_exp2(fmaf(p.sink_v[head], LOG2E, -m * unit));
        else if (p.sink) l += fast_exp2(-m * unit);
      }
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      __nv_bfloat16* dst = p.out + ((size_t)(q_begin + tok0 + row / p.g) * p.Hq + head) * VD;
#pragma unroll 1
      for (int h = 0; h < VD / 32; ++h) {
        uint32_t v[32];
        tmem_ld_32(lane_addr + O_COL0 + h * 32, v);
        tmem_ld_wait();
        if (row < rows) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint4 w;
            w.x = pack_bf16(__uint_as_float(v[c]) * inv, __uint_as_float(v[c + 1]) * inv);
            w.y = pack_bf16(__uint_as_float(v[c + 2]) * inv, __uint_as_float(v[c + 3]) * inv);
            w.z = pack_bf16(__uint_as_float(v[c + 4]) * inv, __uint_as_float(v[c + 5]) * inv);
            w.w = pack_bf16(__uint_as_float(v[c + 6]) * inv, __uint_as_float(v[c + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + h * 32 + c) = w;
          }
        }
      }
    }
    tc_fence_before_sync();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// A bf16 tensor [d3][d2][d1][width] (channels contiguous) seen through boxes [1][b2][b1][64] (d3 = 0: three dimensions), 128-byte
// swizzle; elements outside read as zeros.
int map_of(const void* ptr, int width, long long d1, long long d2, long long d3, int b1, int b2, CUtensorMap* out) {
  tc_host::EncodeTiledFn fn = tc_host::encode_fn();
  if (!fn) return gb::fail(GB_CUDA_ERROR, "cuTensorMapEncodeTiled is not available from this driver");
  const int rank = d3 > 0 ? 4 : 3;
  cuuint64_t dims[4] = {(cuuint64_t)width, (cuuint64_t)d1, (cuuint64_t)d2, (cuuint64_t)(d3 > 0 ? d3 : 1)};
  cuuint64_t strides[3] = {(cuuint64_t)width * 2, (cuuint64_t)width * 2 * d1, (cuuint64_t)width * 2 * d1 * d2};
  cuuint32_t box[4] = {64, (cuuint32_t)b1, (cuuint32_t)b2, 1}, estr[4] = {1, 1, 1, 1};
  const CUresult rc = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(ptr), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? GB_OK : gb::fail(GB_CUDA_ERROR, "cuTensorMapEncodeTiled failed with code %d for a capped attention operand", (int)rc);
}

}  // namespace

namespace capped {

// No line by size: from the first row beyond a decode request's on (17 of a CTA's 128) it takes 0.4 to 1.0 of the mma.sync kernel's time, 1.03 at
// worst (us, this against that, 1 / 16 requests of 5 tokens, 32 heads on 8 of 128 channels without a cap: behind nothing 6.3 / 7.6
// against 6.3 / 7.6, behind 2,048 positions 53 / 64 against 66 / 77, behind 8,192 197 / 268 against 244 / 282).
bool tc_takes(const Params& p, long long pages, int R) {
  const bool page_ok = p.page_size == 8 || p.page_size == 16 || p.page_size == 32 || p.page_size == 64;
  return page_ok && pages > 0 && pages < 0x7fffffff && (p.g & (p.g - 1)) == 0 && p.g <= QROWS && p.Hkv <= 65535 && R <= 65535 && p.scale > 0.f &&
         (((uintptr_t)p.q | (uintptr_t)p.k_pool | (uintptr_t)p.v_pool | (uintptr_t)p.out) & 15) == 0 && tc_host::encode_fn() != nullptr;
}

int launch_tc(const Params& p, int T, long long pages, int R, int max_q_len, cudaStream_t stream) {
  CUtensorMap qm, km, vm;
  const int tokens_per_tile = QROWS / p.g;
  int rc = map_of(p.q, HD, p.Hq, T, 0, p.g, tokens_per_tile, &qm);
  if (rc == GB_OK) rc = map_of(p.k_pool, HD, p.page_size, p.Hkv, pages, p.page_size, 1, &km);
  if (rc == GB_OK) rc = map_of(p.v_pool, VD, p.page_size, p.Hkv, pages, p.page_size, 1, &vm);
  if (rc != GB_OK) return rc;
  const bool cap = p.softcap > 0.f, far = p.r1 != nullptr;
  auto kernel = cap ? (far ? capped_tc_kernel<true, true> : capped_tc_kernel<true, false>)
                    : (far ? capped_tc_kernel<false, true> : capped_tc_kernel<false, false>);
  static gb::OncePerDevice configured;
  if (configured.needed()) {
    for (auto k : {capped_tc_kernel<false, false>, capped_tc_kernel<true, false>, capped_tc_kernel<false, true>, capped_tc_kernel<true, true>}) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
      if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "capped_attention_tc: %s", cudaGetErrorString(e));
    }
    configured.done();
  }
  return gb::check_pdl_launch(gb::launch_pdl(kernel, dim3((max_q_len + tokens_per_tile - 1) / tokens_per_tile, p.Hkv, R), dim3(THREADS), SMEM_BYTES,
                                             stream, dim3(1, 1, 1), qm, km, vm, p, (int)pages),
                              "capped_attention_tc");
}

int tc_error_check() { return gb_err::fetch_and_clear(); }
int tc_set_error_sink(int* host_word) { return gb_err::set_sink(host_word); }

}  // namespace capped

#else  // other widths: the mma.sync kernel

namespace capped {
bool tc_takes(const Params&, long long, int) { return false; }
int launch_tc(const Params&, int, long long, int, int, cudaStream_t) {
  return gb::fail(GB_UNSUPPORTED, "capped_attention_tc: widths %d and %d", GB_KEY_DIM, GB_VALUE_DIM);
}
int tc_error_check() { return 0; }
int tc_set_error_sink(int*) { return 0; }
}  // namespace capped

#endif
