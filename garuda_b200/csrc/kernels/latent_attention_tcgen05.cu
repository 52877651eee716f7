// Causal attention over cached latent rows for prompt portions on the fifth-generation tensor cores: what
// latent_attention_mma.cu computes, for one (RANK, ROT) at a time, with both products as tcgen05.mma, accumulators in
// tensor memory and operands by TMA.
//
// A CTA takes 128 consecutive query rows, (token, head) pairs, of a request and walks the request's cached rows 64 at a time.
// A tile of cached rows is both operands' second half: keys (all its channels, contracted) and values (its first RANK channels,
// MN-major), so it is brought into shared memory once: five blocks of 64 channels for rows of 288, 40 KB, three tiles in flight beside
// the queries' 80 KB.
//   warp 0     TMA: the query tile, then the tiles, one box per page and block of 64 channels. Pages that are not there or that
//              lie behind the last key are asked for beyond the pool's end, which fills their rows with zeros.
//   warp 1     one elected lane: S = Q K^T for two tiles ahead, into one of two S buffers; O += P V of the tile whose softmax just ended,
//              P read from the S buffer in tensor memory. O stays in tensor memory to the end.
//   warps 2-5  a thread owns a query row: its 64 scores, the mask on tiles that reach beyond the tile's first position, exp2 with the
//              scale folded in against the running maximum (where it grows for some row of a warp, that warp rescales O), P in
//              bfloat16 over the scores read. A reference that lags behind the maximum would save most of the rescaling (8 us of the
//              prompt below) but round the largest weights, which are powers of two otherwise: for scores that spread over four powers of e
//              the results would be three times as far off before they are rounded themselves.
// What bounds it: the products (18 of 128 x 64 x 16 for the scores, each as long as one of 128 columns, and 4 of 128 x 256 x 16 a tile,
// about 1,800 cycles), which the softmax of one group of 128 threads fits under; tiles of 128 keys would halve the scores' products but
// not leave room for two of them. A prompt of 2,048 tokens,
// 32 heads over rows of 256 + 32 channels: 350 us with mma.sync, 97 here (calls in a row; 103 before products were issued by an elected lane).
// Every wait is bounded; a wait that runs out sets the error word and the CTA winds down.
#include "error_word.cuh"
#include "tc_common.cuh"
#include "tc_host.cuh"

#if !defined(GB_LATENT_RANK) || !defined(GB_LATENT_ROT)
#error "compile with -DGB_LATENT_RANK=<rank> -DGB_LATENT_ROT=<rot>"
#endif

// whole blocks of 64 value channels, an accumulator that leaves room for the scores
#if GB_LATENT_RANK % 64 == 0 && GB_LATENT_RANK <= 256 && (GB_LATENT_RANK + GB_LATENT_ROT) % 16 == 0 && GB_LATENT_RANK + GB_LATENT_ROT <= 320

namespace {

using namespace tc;

constexpr int RANK = GB_LATENT_RANK, ROW = RANK + GB_LATENT_ROT;
constexpr int BLOCKS = (ROW + 63) / 64, VBLOCKS = RANK / 64;     // blocks of 64 channels: one swizzled 128-byte row each
constexpr int QROWS = 128, KT = 64;
constexpr int ROW_BYTES = 128;
constexpr int Q_BLOCK = QROWS * ROW_BYTES, K_BLOCK = KT * ROW_BYTES;
constexpr int Q_BYTES = BLOCKS * Q_BLOCK, K_BYTES = BLOCKS * K_BLOCK;
constexpr int STAGES = 3, S_BUFS = 2;
constexpr int TILE_BYTES = Q_BYTES + STAGES * K_BYTES;
constexpr int S_COL0 = RANK, TMEM_COLS = 512;
constexpr int THREADS = 64 + QROWS;
static_assert(S_COL0 + S_BUFS * KT <= TMEM_COLS, "tensor memory layout");

struct Misc {
  uint64_t q_full, k_full[STAGES], k_empty[STAGES], s_ready[S_BUFS], p_ready[S_BUFS], o_ready;
  uint32_t tmem_base;
  int abort;
};
constexpr int SMEM_BYTES = TILE_BYTES + (int)sizeof(Misc);
static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void st_shared_zero(uint32_t addr) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(0u) : "memory");
}

// grid (query tiles of the longest request, R)
__global__ void __launch_bounds__(THREADS, 1)
latent_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map, __nv_bfloat16* __restrict__ out,
                 const int32_t* __restrict__ block_table, int table_width, const int32_t* __restrict__ cu_q,
                 const int32_t* __restrict__ kv_lens, int H, float scale_log2, int page_size, int pages, const float* __restrict__ sink_v) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Misc& mc = *reinterpret_cast<Misc*>(smem_raw + TILE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t q_s = smem_u32(smem_raw), k_s = q_s + Q_BYTES;
  if ((q_s & 1023u) != 0) {                                        // the swizzle needs it; never seen
    if (threadIdx.x == 0) gb_err::report(ERR_WAIT_DRAIN);
    return;
  }
  const int r = blockIdx.y;
  // The batch's lengths and tables were copied in before the step's first kernel.
  const int q_begin = cu_q[r], q_len = cu_q[r + 1] - q_begin, kv_len = kv_lens[r];
  const int row0 = (int)(gridDim.x - 1 - blockIdx.x) * QROWS;      // the last rows, which read the most keys, first
  const int rows = min(QROWS, q_len * H - row0);
  if (rows <= 0) return;
  const int pos0 = kv_len - q_len;
  const int hi = pos0 + (row0 + rows - 1) / H;                     // the last key that a row of the tile reads
  const int n_tiles = hi / KT + 1;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&mc.q_full), 1);
    mbar_init(smem_u32(&mc.o_ready), 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&mc.k_full[s]), 1);
      mbar_init(smem_u32(&mc.k_empty[s]), 1);
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
  gb::pdl_wait();      // queries and this step's rows come from the kernels in front

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA
    const int per_tile = KT / page_size;                           // 1 to 8 pages, a lane each
    const int32_t* table = block_table + (size_t)r * table_width;
    int loaded = 0;                                                // tiles asked for
    if (lane == 0) {
      mbar_arrive_expect_tx(smem_u32(&mc.q_full), Q_BYTES);
#pragma unroll
      for (int b = 0; b < BLOCKS; ++b) tma_load_2d(q_s + b * Q_BLOCK, &q_map, smem_u32(&mc.q_full), b * 64, q_begin * H + row0);
    }
    for (int t = 0; t < n_tiles; ++t) {
      const int st = t % STAGES;
      const int first = t * KT + lane * page_size;
      int page = lane < per_tile && first <= hi ? table[first / page_size] : -1;
      if (page < 0 || page >= pages) page = pages;                 // beyond the pool: zeros
      if (lane == 0) {
        if (t >= STAGES && !mbar_wait(smem_u32(&mc.k_empty[st]), (t / STAGES - 1) & 1)) {
          gb_err::report(ERR_WAIT_EMPTY);
          *abort_s = 1;
        }
        if (!*abort_s) mbar_arrive_expect_tx(smem_u32(&mc.k_full[st]), K_BYTES);
      }
      __syncwarp();
      if (*abort_s) break;
      if (lane < per_tile) {
#pragma unroll
        for (int b = 0; b < BLOCKS; ++b)
          tma_load_3d(k_s + st * K_BYTES + b * K_BLOCK + lane * page_size * ROW_BYTES, &k_map, smem_u32(&mc.k_full[st]), b * 64, 0, page);
      }
      loaded = t + 1;
    }
    // wind down, or just end: the copies in flight land before the CTA's shared memory is given up
    if (lane == 0) {
      bool ok = mbar_wait(smem_u32(&mc.q_full), 0);
      for (int t = loaded > STAGES ? loaded - STAGES : 0; t < loaded; ++t) ok = mbar_wait(smem_u32(&mc.k_full[t % STAGES]), (t / STAGES) & 1) && ok;
      if (!ok) gb_err::report(ERR_WAIT_DRAIN);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issuer
    const bool leader = elect_one();
    constexpr uint32_t idesc_s = instr_desc_bf16(QROWS, KT);
    constexpr uint32_t idesc_o = instr_desc_bf16(QROWS, RANK) | INSTR_B_MN_MAJOR;
    const uint64_t dq0 = smem_desc_sw128(q_s), dk0 = smem_desc_sw128(k_s), dv0 = smem_desc_sw128_mn(k_s, K_BLOCK);
    bool ok = mbar_wait(smem_u32(&mc.q_full), 0);
    if (!ok && lane == 0) gb_err::report(ERR_WAIT_FULL);
    auto issue_s = [&](int t) {
      const int st = t % STAGES, buf = t % S_BUFS;
      if (!mbar_wait(smem_u32(&mc.k_full[st]), (t / STAGES) & 1)) {
        if (lane == 0) gb_err::report(ERR_WAIT_FULL);
        ok = false;
        return;
      }
      tc_fence_after_sync();
      if (leader) {
#pragma unroll
        for (int k = 0; k < ROW / 16; ++k)                         // 16 channels a product, 32 bytes on within a block's rows
          mma_bf16(tmem_base + S_COL0 + buf * KT, dq0 + (uint64_t)((k / 4) * (Q_BLOCK >> 4) + (k % 4) * 2),
                   dk0 + (uint64_t)(st * (K_BYTES >> 4) + (k / 4) * (K_BLOCK >> 4) + (k % 4) * 2), idesc_s, k > 0);
        mma_commit(smem_u32(&mc.s_ready[buf]));
      }
      __syncwarp();
    };
    for (int t = 0; t < S_BUFS && t < n_tiles && ok; ++t) issue_s(t);
    for (int t = 0; t < n_tiles && ok; ++t) {
      const int st = t % STAGES, buf = t % S_BUFS;
      if (*abort_s) break;
      if (!mbar_wait(smem_u32(&mc.p_ready[buf]), (t / S_BUFS) & 1)) {
        if (lane == 0) gb_err::report(ERR_WAIT_ACCUM);
        ok = false;
        break;
      }
      tc_fence_after_sync();
      if (leader) {
        mma_bf16_ts<KT / 16>(tmem_base, tmem_base + S_COL0 + buf * KT, dv0 + (uint64_t)(st * (K_BYTES >> 4)), idesc_o, 16 * ROW_BYTES >> 4, t > 0);
        mma_commit(smem_u32(&mc.k_empty[st]));
        mma_commit(smem_u32(&mc.o_ready));
      }
      __syncwarp();
      // the products above read their P from this buffer before the next one writes (products run in the order of their issue)
      if (t + S_BUFS < n_tiles) issue_s(t + S_BUFS);
    }
    if (!ok) *abort_s = 1;
  } else {
    // -------------------------------------------------------------------- softmax warps
    const int quarter = warp & 3;                                  // the TMEM lanes this warp may read
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int row_pos = row < rows ? pos0 + (row0 + row) / H : -1; // no key is valid for a padding row
    const int first_pos = pos0 + row0 / H;
    float m = -INFINITY, l = 0.f;                                  // m: the largest raw dot product so far
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
      const uint32_t s_addr = lane_addr + S_COL0 + buf * KT;
      uint32_t sv[KT / 32][32];
#pragma unroll
      for (int h = 0; h < KT / 32; ++h) tmem_ld_32(s_addr + h * 32, sv[h]);
      const int key0 = t * KT;
      if (key0 + KT - 1 > hi) {
        // Rows behind the last key are the unwritten end of a page: their probabilities are zero, but zero times a stray NaN is
        // not. (The scores' products have read the stage; the values' ones do so after this thread's arrival below.)
        if (row < KT && key0 + row > hi) {
#pragma unroll
          for (int b = 0; b < VBLOCKS; ++b)
#pragma unroll
            for (int c = 0; c < ROW_BYTES / 16; ++c) st_shared_zero(k_s + st * K_BYTES + b * K_BLOCK + row * ROW_BYTES + c * 16);
        }
        fence_proxy_async();
      }
      tmem_ld_wait();
      auto sc = [&](int c) -> float& { return reinterpret_cast<float&>(sv[c >> 5][c & 31]); };
      if (key0 + KT - 1 > first_pos) {
#pragma unroll
        for (int c = 0; c < KT; ++c)
          if (key0 + c > row_pos) sc(c) = -INFINITY;
      }
      float mx[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < KT; c += 4)
#pragma unroll
        for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], sc(c + e));
      const float m_new = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      const bool grown = m != -INFINITY && m_new > m;
      bool waited = false;
      if (t > 0 && __any_sync(0xffffffffu, grown)) {
        wait_o(t - 1);
        waited = true;
        if (!ok) break;
        const float corr = m == -INFINITY ? 1.f : fast_exp2((m - m_new) * scale_log2);
#pragma unroll 1
        for (int h = 0; h < RANK; h += 64) {
          uint32_t v[2][32];
          tmem_ld_32(lane_addr + h, v[0]);
          tmem_ld_32(lane_addr + h + 32, v[1]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 64; ++c) v[c >> 5][c & 31] = __float_as_uint(__uint_as_float(v[c >> 5][c & 31]) * corr);
          tmem_st_32(lane_addr + h, v[0]);
          tmem_st_32(lane_addr + h + 32, v[1]);
        }
        l *= corr;
        m = m_new;
      } else if (m == -INFINITY) {
        m = m_new;
      }
      const float neg_m = m == -INFINITY ? 0.f : -m * scale_log2;  // nothing valid yet: avoid inf - inf
#pragma unroll
      for (int c = 0; c < KT; ++c) sc(c) = fast_exp2(fmaf(sc(c), scale_log2, neg_m));
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[KT / 2];
#pragma unroll
      for (int c = 0; c < KT; c += 2) {
        // (the denominator counts the weights as they are multiplied: their rounding then cancels in part)
        pk[c >> 1] = pack_bf16(sc(c), sc(c + 1));
        ls[(c >> 1) & 3] += __uint_as_float(pk[c >> 1] << 16) + __uint_as_float(pk[c >> 1] & 0xffff0000u);
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
      // a learned sink per head: exp(sink_h) in the denominator, without a key or a value
      if (sink_v != nullptr && m != -INFINITY) l += fast_exp2(sink_v[(row0 + row) % H] * 1.4426950408889634f - m * scale_log2);
      const float inv = l > 0.f ? 1.0f / l : 0.f;
      __nv_bfloat16* dst = out + ((size_t)q_begin * H + row0 + row) * RANK;
#pragma unroll 1
      for (int h = 0; h < RANK / 32; ++h) {
        uint32_t v[32];
        tmem_ld_32(lane_addr + h * 32, v);
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

// The pool [pages][page_size][ROW] through boxes of a page by 64 channels, 128-byte swizzle; what lies outside reads as zeros.
int pool_map(const void* pool, int pages, int page_size, CUtensorMap* out) {
  tc_host::EncodeTiledFn fn = tc_host::encode_fn();
  if (!fn) return gb::fail(GB_CUDA_ERROR, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[3] = {(cuuint64_t)ROW, (cuuint64_t)page_size, (cuuint64_t)pages};
  cuuint64_t strides[2] = {(cuuint64_t)ROW * 2, (cuuint64_t)ROW * 2 * page_size};
  cuuint32_t box[3] = {64, (cuuint32_t)page_size, 1}, estr[3] = {1, 1, 1};
  const CUresult rc = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(pool), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? GB_OK : gb::fail(GB_CUDA_ERROR, "cuTensorMapEncodeTiled failed with code %d for a latent pool", (int)rc);
}

}  // namespace

// Whether the kernel takes these sizes and addresses.
GB_EXPORT int gb_latent_attention_tc_takes(const void* q, const void* pool, const void* out, int page_size, int pages, long long rows) {
  const bool page_ok = page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64;
  return page_ok && pages > 0 && rows > 0 && rows < 0x7fffffffLL && (((uintptr_t)q | (uintptr_t)pool | (uintptr_t)out) & 15) == 0 &&
         tc_host::encode_fn() != nullptr;
}

// q [T, H, ROW], pool [pages, 1, page_size, ROW], out [T, H * RANK], all bfloat16; the rest as gb_latent_attention.
GB_EXPORT int gb_latent_attention_tc(const void* q, const void* pool, void* out, const int32_t* block_table, int table_width,
                                     const int32_t* cu_q, const int32_t* kv_lens, int T, int num_requests, int H, float scale,
                                     int page_size, int pages, int max_q_len, const float* sink_v, cudaStream_t stream) {
  if (T <= 0 || num_requests <= 0) return GB_OK;
  if (H < 1 || max_q_len < 1 || num_requests > 65535 || !(scale > 0.f) || !gb_latent_attention_tc_takes(q, pool, out, page_size, pages, (long long)T * H))
    return gb::fail(GB_UNSUPPORTED, "latent_attention_tc: heads %d, page size %d, %d pages, scale %g", H, page_size, pages, (double)scale);
  CUtensorMap qm, km;
  int rc = tc_host::tensor_map_2d(q, (long long)T * H, ROW, QROWS, &qm);
  if (rc != GB_OK) return rc;
  rc = pool_map(pool, pages, page_size, &km);
  if (rc != GB_OK) return rc;
  static gb::OncePerDevice configured;
  if (configured.needed()) {
    const cudaError_t e = cudaFuncSetAttribute(latent_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "latent_attention_tc: %s", cudaGetErrorString(e));
    configured.done();
  }
  const long long tiles = ((long long)max_q_len * H + QROWS - 1) / QROWS;
  return gb::check_pdl_launch(gb::launch_pdl(latent_tc_kernel, dim3((unsigned)tiles, num_requests), dim3(THREADS), SMEM_BYTES, stream,
                                             dim3(1, 1, 1), qm, km, (__nv_bfloat16*)out, block_table, table_width, cu_q, kv_lens, H,
                                             scale * 1.4426950408889634f, page_size, pages, sink_v),
                              "latent_attention_tc");
}

GB_EXPORT int gb_latent_attention_error_check() { return gb_err::fetch_and_clear(); }
GB_EXPORT int gb_latent_attention_set_error_sink(int* host_word) { return gb_err::set_sink(host_word); }

#else  // other sizes: the mma.sync kernel

GB_EXPORT int gb_latent_attention_tc_takes(const void*, const void*, const void*, int, int, long long) { return 0; }
GB_EXPORT int gb_latent_attention_tc(const void*, const void*, void*, const int32_t*, int, const int32_t*, const int32_t*, int, int, int, float,
                                     int, int, int, const float*, cudaStream_t) {
  return gb::fail(GB_UNSUPPORTED, "latent_attention_tc: latent %d + %d", GB_LATENT_RANK, GB_LATENT_ROT);
}
GB_EXPORT int gb_latent_attention_error_check() { return 0; }
GB_EXPORT int gb_latent_attention_set_error_sink(int*) { return 0; }

#endif
