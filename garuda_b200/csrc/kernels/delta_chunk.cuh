// A delta-rule recurrence walked a chunk of 32 tokens at a time instead of token by token: the serial half,
// shared by the gated rule (delta_rule.cu) and the generalized one (general_delta.cu).
//
// Within a chunk that starts from the state S [dim, vdim], with D_i the product of the tokens' decays up to i,
// both rules are linear in S once a small triangular system per chunk has been solved, which needs the chunk's
// keys, queries and decays only (the form of Yang et al., "Parallelizing Linear Transformers with the Delta Rule
// over Sequence Length", 2024). A kernel in front of this one, a block per (chunk, head), leaves for every chunk
//     WQ [2 C, dim]   the rows W_i, then Q_i
//     K1 [C, dim]     what a token's row Y_i is written with, decayed to the chunk's end;  (K2 [C, dim] likewise for
//                     a second, known row V_i: the generalized rule)
//     last [dim]      the chunk's whole decay
//     VP, OP [C, vdim] (and V [C, vdim])
// and this one walks a request's chunks in order:
//     Y = VP - W S;   o = OP + Q S;   S <- diag(last) S + K1^T Y (+ K2^T V)
//
// The products run on the tensor cores (mma.sync m16n8k8, tf32 operands, 32-bit sums) with every 32-bit
// operand as the sum of two tf32 numbers, which hold 22 of its 24 bits; three products (the low parts'
// own is left out) are added up. The state itself stays in 32-bit registers from the request's first token of the step to
// its last, and the tensor cores' sums, which are cut off and not rounded, are of eight products only: those pieces, and a
// chunk's update of the state, are added by rounded 32-bit operations. With sums of 32 products in the tensor cores the read-outs and the
// state of 2,048 tokens were 1.2 to 1.4 times as far from 64 bits as the token-by-token kernels' where decays forget within some tens of tokens;
// now 0.7 to 1.1 times, at 237 us against 234 for the channel rule's kernels.
//
// Why this split: the token-by-token kernels are bound by a token's chain of dependent sums and shuffles (0.43 us a
// token of 16 heads of 128 x 128, whatever the tokens do); a chunk's three products have no chain. On multiply-adds instead of the
// tensor cores the walk was bound by shared memory, whose bandwidth serves four multiply-adds a number only (162 us for 2,048 tokens).
// A group of four warps has 16 columns of S, a quarter of the channels each: S^T in the accumulators' layout is at once the first
// operand of S^T [W; Q]^T, so nothing of S is ever exchanged, only the warps' shares of Y and o. One group a block while the
// walked requests' blocks are at most one an SM (16 heads x 8 groups are 128 blocks for 148 SMs); two (which share WQ, K1 and K2) where the
// heads are more. 2,048 tokens of 16 heads of 128 x 128 take 98 us here and 119 us in the kernel in front (B200), where the
// token-by-token walk took 0.89 ms; the tensor cores are 44% busy, the rest is the latency of a chunk's three barriers.
#pragma once

#include "common.cuh"

namespace delta_chunk {

constexpr int C = 32;              // tokens of a chunk
constexpr int COLS = 16;           // columns of S of a group of four warps
constexpr int GROUP = 128;         // threads of a group

// Floats of a chunk's block for one head. The first `staged` of them go through shared memory. WQ and K1 (K2) lie in tiles of
// 8 x 8 numbers, in the order in which the products' second operands are read; VP, OP and V lie column by column.
struct Layout {
  int dim, vdim, two;
  __host__ __device__ int staged() const { return dim * 2 * C + C * dim * (1 + two) + dim; }
  __host__ __device__ int k1() const { return dim * 2 * C; }
  __host__ __device__ int last() const { return k1() + C * dim * (1 + two); }
  __host__ __device__ int vp() const { return staged(); }
  __host__ __device__ int op() const { return vp() + C * vdim; }
  __host__ __device__ int v() const { return op() + C * vdim; }
  __host__ __device__ int floats() const { return v() + (two ? C * vdim : 0); }
  // row i of W (C + i: of Q), channel c: tiles of 8 rows x 8 channels, a row's channels together
  __host__ __device__ int wq(int row, int c) const { return ((c >> 3) * (2 * C / 8) + (row >> 3)) * 64 + (row & 7) * 8 + (c & 7); }
  // token j, channel c of K1: tiles of 8 channels x 8 tokens, a channel's tokens together
  __host__ __device__ int k1(int j, int c) const { return k1() + ((j >> 3) * (dim / 8) + (c >> 3)) * 64 + (c & 7) * 8 + (j & 7); }
};

// Chunks are numbered over the requests that are walked (of `cut` tokens or more in the step), so that no two share a number and a
// step's many short requests take no room: the chunks of the w-th of them (from 0), which starts at token t0, have the numbers from
// t0 / C + w on. All numbers of `walked` such requests are below chunk_numbers(T, walked).
__host__ __device__ __forceinline__ int chunk_numbers(int T, int walked) { return T / C + walked; }

// The w-th request that is walked (all threads of a warp call this); -1: there are no more.
__device__ __forceinline__ int nth_walked(const int32_t* __restrict__ cu_q, int R, int cut, int w) {
  const int lane = threadIdx.x & 31;
  for (int r0 = 0; r0 < R; r0 += 32) {
    const int r = min(r0 + lane, R - 1);
    const uint32_t walked = __ballot_sync(0xffffffffu, r0 + lane < R && cu_q[r + 1] - cu_q[r] >= cut);
    const uint32_t it = __ballot_sync(0xffffffffu, (walked >> lane & 1) && __popc(walked & ((1u << lane) - 1)) == w);
    if (it != 0) return r0 + __ffs(it) - 1;
    w -= __popc(walked);
  }
  return -1;
}

// The request and chunk of a number (all threads of a warp call this): false where there is none.
__device__ __forceinline__ bool find_chunk(int number, const int32_t* __restrict__ cu_q, int R, int cut, int& request, int& first,
                                           int& tokens, int& in_request) {
  const int lane = threadIdx.x & 31;
  int count = 0, best = -1, start = 0;       // the last walked request whose first number is not above this one, and that first number
  for (int r0 = 0; r0 < R; r0 += 32) {
    const int r = min(r0 + lane, R - 1), t0 = cu_q[r];
    const uint32_t walked = __ballot_sync(0xffffffffu, r0 + lane < R && cu_q[r + 1] - t0 >= cut);
    const int at = t0 / C + count + __popc(walked & ((1u << lane) - 1));
    if ((walked >> lane & 1) && at <= number) best = r, start = at;
    count += __popc(walked);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {         // both grow with the request
    best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    start = max(start, __shfl_xor_sync(0xffffffffu, start, o));
  }
  if (best < 0) return false;
  const int t0 = cu_q[best], n = cu_q[best + 1] - t0;
  in_request = (number - start) * C;
  if (in_request >= n) return false;
  request = best, first = t0 + in_request, tokens = min(C, n - in_request);
  return true;
}

// ---- two 32-bit multiply-adds in one instruction -----------------------------------------------
using pair_t = unsigned long long;
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
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
  pair_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ pair_t mul2(pair_t a, pair_t b) {
  pair_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
struct __align__(16) pair2_t { pair_t a, b; };

// The sums over a warp of eight values: lane l gets the sum of value l / 4.
__device__ __forceinline__ float sum_of_eight(float (&v)[8], int lane) {
#pragma unroll
  for (int half = 4; half > 0; half >>= 1) {
    const bool upper = lane & (half * 4);
#pragma unroll
    for (int x = 0; x < half; ++x) {
      const float give = upper ? v[x] : v[x + half], mine = upper ? v[x + half] : v[x];
      v[x] = mine + __shfl_xor_sync(0xffffffffu, give, half * 4);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// ---- the substitution's building blocks: a column of C numbers in registers, in pairs -----------
constexpr int LT = C + 4;            // floats between the rows of the small matrices

// x_i += sign * m[j][i] * y for the i > j (STRICT) or i >= j; m is held transposed, a row per j. Numbers of the other
// side of the diagonal are not touched: an infinity at token j must not reach the tokens in front of it.
template <bool STRICT>
__device__ __forceinline__ void add_row(pair_t (&x)[C / 2], const float* m, int j, float y) {
  const int from = STRICT ? j + 1 : j;
  const pair_t yy = make_pair(y, y);
#pragma unroll
  for (int i4 = 0; i4 < C; i4 += 4) {
    if (i4 + 3 < from) continue;
    const pair2_t f = *reinterpret_cast<const pair2_t*>(m + j * LT + i4);
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int i = i4 + 2 * p;
      const pair_t c = p ? f.b : f.a;
      if (i >= from) {
        x[i / 2] = fma2(c, yy, x[i / 2]);
      } else if (i + 1 >= from) {
        const float2 old = both(x[i / 2]);
        x[i / 2] = make_pair(old.x, fmaf(both(c).y, y, old.y));
      }
    }
  }
}
__device__ __forceinline__ float entry(const pair_t (&x)[C / 2], int i) { return i & 1 ? both(x[i / 2]).y : both(x[i / 2]).x; }
__device__ __forceinline__ void set_entry(pair_t (&x)[C / 2], int i, float v) {
  const float2 old = both(x[i / 2]);
  x[i / 2] = i & 1 ? make_pair(old.x, v) : make_pair(v, old.y);
}

__device__ __forceinline__ void store_rows(float* block, const Layout& lay, int first_row, int c, const pair_t (&x)[C / 2]) {
#pragma unroll
  for (int i = 0; i < C; ++i) block[lay.wq(first_row + i, c)] = entry(x, i);
}
__device__ __forceinline__ void store_column(float* to, const pair_t (&x)[C / 2]) {
#pragma unroll
  for (int i = 0; i < C / 4; ++i) {
    const float2 a = both(x[2 * i]), b = both(x[2 * i + 1]);
    reinterpret_cast<float4*>(to)[i] = make_float4(a.x, a.y, b.x, b.y);
  }
}

// ---- the walk ------------------------------------------------------------------------------------
__device__ __forceinline__ void copy_16(float* smem, const float* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}

// A 32-bit number as two tf32 ones: the nearest (ties away from zero), and the rest, whose low bits the tensor cores do
// not read (the rest has either sign, so cutting it off leans to neither side). A number that is not finite makes the rest not a
// number, whatever the rounding makes of its own bits.
__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_1688(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the same with nothing added
__device__ __forceinline__ void mma_1688_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

constexpr int LDR = 2 * C + 8, LDY = C + 8;        // floats between columns in shared memory: eight columns' reads fall into different banks

template <int DIM, int GROUPS, bool TWO>
struct WalkSmem {
  float stage[2][DIM * 2 * C + C * DIM * (TWO ? 2 : 1) + DIM];
  float red[GROUPS][4][COLS][LDR];         // the warps' shares of (W S)^T and (Q S)^T
  float y[GROUPS][TWO ? 2 : 1][COLS][LDY]; // Y^T (and V^T)
};

// grid (H, vdim / (16 GROUPS), walked): a block for a request that is not walked would hold an SM's shared memory only to return (64 single
// tokens beside a prompt of 48, 16 heads: 152 us, with blocks for all 167). blocks [numbers, H, Layout::floats()]. out [T, H vdim].
template <int DIM, int GROUPS, bool TWO>
__global__ void __launch_bounds__(GROUP * GROUPS, 1)
walk_kernel(const float* __restrict__ blocks, const int32_t* __restrict__ cu_q, const int32_t* __restrict__ slots,
            float* __restrict__ state, long long state_stride, int R, int H, int vdim, int cut, int numbers, float* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char raw[];
  using Smem = WalkSmem<DIM, GROUPS, TWO>;
  Smem& sm = *reinterpret_cast<Smem*>(raw);
  gb::pdl_wait();
  const int h = blockIdx.x, r = nth_walked(cu_q, R, cut, blockIdx.z);
  if (r < 0) return;
  const int t0 = cu_q[r], n = cu_q[r + 1] - t0, number = t0 / C + blockIdx.z;
  const Layout lay{DIM, vdim, TWO ? 1 : 0};
  constexpr int THREADS = GROUP * GROUPS;
  constexpr int KS = DIM / 32;                       // tiles of 8 channels of a warp
  const int grp = threadIdx.x / GROUP, tid = threadIdx.x % GROUP, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, tig = lane & 3;
  const int col0 = (blockIdx.y * GROUPS + grp) * COLS;
  const int mycol = (tid >> 1) & 15, tok4 = ((tid & 1) | (warp << 1)) * 4;      // where Y and o are formed: a column, four tokens
  const int slot = slots[r];
  const int chunks = (n + C - 1) / C;
  if (number + chunks > numbers) return;             // more requests than the caller counted: nothing beyond blocks is read
  const size_t per = (size_t)H * lay.floats();
  const float* base = blocks + ((size_t)number * H + h) * lay.floats();

  auto load = [&](int k) {
    const float* src = base + k * per;
    float* dst = sm.stage[k & 1];
    for (int i = threadIdx.x * 4; i < (int)(sizeof(sm.stage[0]) / 4); i += THREADS * 4) copy_16(dst + i, src + i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // S^T in accumulator tiles of 16 columns x 8 channels: S[m][e] is column g + 8 (e / 2), channel 2 tig + (e & 1) of tile m
  float* S_g = slot >= 0 ? state + (size_t)slot * state_stride + (size_t)h * DIM * vdim + col0 : nullptr;
  const int ch0 = warp * (DIM / 4) + 2 * tig;
  float S[KS][4];
#pragma unroll
  for (int m = 0; m < KS; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) S[m][e] = S_g ? S_g[(size_t)(ch0 + m * 8 + (e & 1)) * vdim + g + 8 * (e >> 1)] : 0.f;
  const float* columns = base + (size_t)(col0 + mycol) * C + tok4;
  load(0);
  float4 vp = *reinterpret_cast<const float4*>(columns + lay.vp());
  float4 op = *reinterpret_cast<const float4*>(columns + lay.op());
  float4 vv = make_float4(0.f, 0.f, 0.f, 0.f);
  if (TWO) vv = *reinterpret_cast<const float4*>(columns + lay.v());
  for (int k = 0; k < chunks; ++k) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                // this chunk has landed; everyone is done with the chunk in front
    if (k + 1 < chunks) load(k + 1);
    const float* stage = sm.stage[k & 1];
    // ---- this warp's channels of (W S)^T and (Q S)^T. The eight channels of a step are taken in the order in which the
    // accumulators hold them: places tig and tig + 4 are channels 2 tig and 2 tig + 1
    {
      float acc[2 * C / 8][4];
#pragma unroll
      for (int i = 0; i < 2 * C / 8; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
      const float* b = stage + warp * KS * (2 * C / 8) * 64 + lane * 2;
#pragma unroll
      for (int m = 0; m < KS; ++m) {
        uint32_t hi[4], lo[4];
        split(S[m][0], hi[0], lo[0]), split(S[m][2], hi[1], lo[1]), split(S[m][1], hi[2], lo[2]), split(S[m][3], hi[3], lo[3]);
        uint32_t bh[2 * C / 8][2], bl[2 * C / 8][2];
#pragma unroll
        for (int i = 0; i < 2 * C / 8; ++i) {
          const float2 f = *reinterpret_cast<const float2*>(b + (m * (2 * C / 8) + i) * 64);
          split(f.x, bh[i][0], bl[i][0]), split(f.y, bh[i][1], bl[i][1]);
        }
        float piece[2 * C / 8][4];
#pragma unroll
        for (int i = 0; i < 2 * C / 8; ++i) mma_1688_first(piece[i], lo, bh[i][0], bh[i][1]);
#pragma unroll
        for (int i = 0; i < 2 * C / 8; ++i) mma_1688(piece[i], hi, bl[i][0], bl[i][1]);
#pragma unroll
        for (int i = 0; i < 2 * C / 8; ++i) mma_1688(piece[i], hi, bh[i][0], bh[i][1]);
#pragma unroll
        for (int i = 0; i < 2 * C / 8; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][e] += piece[i][e];
      }
#pragma unroll
      for (int i = 0; i < 2 * C / 8; ++i) {
        *reinterpret_cast<float2*>(&sm.red[grp][warp][g][i * 8 + 2 * tig]) = make_float2(acc[i][0], acc[i][1]);
        *reinterpret_cast<float2*>(&sm.red[grp][warp][g + 8][i * 8 + 2 * tig]) = make_float2(acc[i][2], acc[i][3]);
      }
    }
    __syncthreads();
    // ---- Y = VP - W S, o = OP + Q S
    {
      float4 part[2][4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        part[0][w] = *reinterpret_cast<const float4*>(&sm.red[grp][w][mycol][tok4]);
        part[1][w] = *reinterpret_cast<const float4*>(&sm.red[grp][w][mycol][C + tok4]);
      }
      auto sum = [](float a, float b, float c, float d) { return (a + b) + (c + d); };
      float4 y, o;
      y.x = vp.x - sum(part[0][0].x, part[0][1].x, part[0][2].x, part[0][3].x), y.y = vp.y - sum(part[0][0].y, part[0][1].y, part[0][2].y, part[0][3].y);
      y.z = vp.z - sum(part[0][0].z, part[0][1].z, part[0][2].z, part[0][3].z), y.w = vp.w - sum(part[0][0].w, part[0][1].w, part[0][2].w, part[0][3].w);
      o.x = op.x + sum(part[1][0].x, part[1][1].x, part[1][2].x, part[1][3].x), o.y = op.y + sum(part[1][0].y, part[1][1].y, part[1][2].y, part[1][3].y);
      o.z = op.z + sum(part[1][0].z, part[1][1].z, part[1][2].z, part[1][3].z), o.w = op.w + sum(part[1][0].w, part[1][1].w, part[1][2].w, part[1][3].w);
      *reinterpret_cast<float4*>(&sm.y[grp][0][mycol][tok4]) = y;
      if (TWO) *reinterpret_cast<float4*>(&sm.y[grp][TWO ? 1 : 0][mycol][tok4]) = vv;
      const int t = k * C + tok4;
      float* to = out + (size_t)(t0 + t) * H * vdim + h * vdim + col0 + mycol;
      const size_t row = (size_t)H * vdim;
      if (t < n) to[0] = o.x;
      if (t + 1 < n) to[row] = o.y;
      if (t + 2 < n) to[2 * row] = o.z;
      if (t + 3 < n) to[3 * row] = o.w;
    }
    if (k + 1 < chunks) {
      columns += per;
      vp = *reinterpret_cast<const float4*>(columns + lay.vp());
      op = *reinterpret_cast<const float4*>(columns + lay.op());
      if (TWO) vv = *reinterpret_cast<const float4*>(columns + lay.v());
    }
    __syncthreads();                // Y is whole
    // ---- S <- diag(last) S + K1^T Y (+ K2^T V); tokens in the same order of places
    {
      float acc[KS][4];
#pragma unroll
      for (int m = 0; m < KS; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][e] = 0.f;
#pragma unroll
      for (int part = 0; part < (TWO ? 2 : 1); ++part) {
        const float* b = stage + lay.k1() + part * C * DIM + warp * KS * 64 + lane * 2;
#pragma unroll
        for (int j = 0; j < C / 8; ++j) {
          const float2 y0 = *reinterpret_cast<const float2*>(&sm.y[grp][part][g][j * 8 + 2 * tig]);
          const float2 y1 = *reinterpret_cast<const float2*>(&sm.y[grp][part][g + 8][j * 8 + 2 * tig]);
          uint32_t hi[4], lo[4];
          split(y0.x, hi[0], lo[0]), split(y1.x, hi[1], lo[1]), split(y0.y, hi[2], lo[2]), split(y1.y, hi[3], lo[3]);
          uint32_t bh[KS][2], bl[KS][2];
#pragma unroll
          for (int m = 0; m < KS; ++m) {
            const float2 f = *reinterpret_cast<const float2*>(b + (j * (DIM / 8) + m) * 64);
            split(f.x, bh[m][0], bl[m][0]), split(f.y, bh[m][1], bl[m][1]);
          }
          float piece[KS][4];
#pragma unroll
          for (int m = 0; m < KS; ++m) mma_1688_first(piece[m], lo, bh[m][0], bh[m][1]);
#pragma unroll
          for (int m = 0; m < KS; ++m) mma_1688(piece[m], hi, bl[m][0], bl[m][1]);
#pragma unroll
          for (int m = 0; m < KS; ++m) mma_1688(piece[m], hi, bh[m][0], bh[m][1]);
#pragma unroll
          for (int m = 0; m < KS; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[m][e] += piece[m][e];
        }
      }
#pragma unroll
      for (int m = 0; m < KS; ++m) {
        const float2 whole = *reinterpret_cast<const float2*>(stage + lay.last() + ch0 + m * 8);
#pragma unroll
        for (int e = 0; e < 4; ++e) S[m][e] = fmaf(e & 1 ? whole.y : whole.x, S[m][e], acc[m][e]);
      }
    }
  }
  // only now may the next kernel in the stream start: its blocks would wait beside these for the whole walk
  gb::pdl_launch_dependents();
  if (S_g != nullptr) {
#pragma unroll
    for (int m = 0; m < KS; ++m)
#pragma unroll
      for (int e = 0; e < 4; ++e) S_g[(size_t)(ch0 + m * 8 + (e & 1)) * vdim + g + 8 * (e >> 1)] = S[m][e];
  }
}

template <int DIM, int GROUPS, bool TWO>
int launch_walk_as(const char* what, const float* blocks, const int32_t* cu_q, const int32_t* slots, float* state, long long state_stride,
                   int R, int walked, int H, int vdim, int cut, int numbers, float* out, cudaStream_t stream) {
  auto kernel = walk_kernel<DIM, GROUPS, TWO>;
  constexpr size_t smem = sizeof(WalkSmem<DIM, GROUPS, TWO>);
  static_assert(smem <= 227 * 1024, "a block's shared memory");
  static gb::OncePerDevice configured;
  if (configured.needed()) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "%s: %s", what, cudaGetErrorString(e));
    configured.done();
  }
  return gb::check_pdl_launch(gb::launch_after(kernel, dim3(H, vdim / (COLS * GROUPS), walked), dim3(GROUP * GROUPS), smem, stream,
                                               dim3(1, 1, 1), blocks, cu_q, slots, state, state_stride, R, H, vdim, cut, numbers, out),
                              what);
}

// dim 64 or 128, vdim a multiple of 32. numbers: what blocks has room for, chunk_numbers(T, walked).
template <bool TWO>
int launch_walk(const char* what, const float* blocks, const int32_t* cu_q, const int32_t* slots, float* state, long long state_stride,
                int R, int walked, int H, int dim, int vdim, int cut, int numbers, float* out, cudaStream_t stream) {
  // requests that are not walked have no blocks to speak of: a prompt of 2,048 tokens beside eight single ones, 379 us, now 294
  const bool one = (long long)walked * H * (vdim / COLS) <= gb::sm_count();
  if (dim == 128)
    return one ? launch_walk_as<128, 1, TWO>(what, blocks, cu_q, slots, state, state_stride, R, walked, H, vdim, cut, numbers, out, stream)
               : launch_walk_as<128, 2, TWO>(what, blocks, cu_q, slots, state, state_stride, R, walked, H, vdim, cut, numbers, out, stream);
  return one ? launch_walk_as<64, 1, TWO>(what, blocks, cu_q, slots, state, state_stride, R, walked, H, vdim, cut, numbers, out, stream)
             : launch_walk_as<64, 2, TWO>(what, blocks, cu_q, slots, state, state_stride, R, walked, H, vdim, cut, numbers, out, stream);
}

inline bool takes(int dim, int vdim) { return (dim == 64 || dim == 128) && vdim >= 32 && vdim % 32 == 0 && vdim <= 256; }

}  // namespace delta_chunk
