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
// by pieces 0.7 to 1.1 times, at 237 us against 234 for the channel rule's kernels.
//
// Why this split: the token-by-token kernels are bound by a token's chain of dependent sums and shuffles (0.43 us a
// token of 16 heads of 128 x 128, whatever the tokens do); a chunk's three products have no chain. On multiply-adds instead of the
// tensor cores the walk was bound by shared memory, whose bandwidth serves four multiply-adds a number only (162 us for 2,048 tokens).
// A group of four warps has 16 columns of S, a quarter of the channels each: S^T in the accumulators' layout is at once the first
// operand of S^T [W; Q]^T, so nothing of S is ever exchanged, only the warps' shares of Y and o. One group a block while the
// walked requests' blocks are at most one an SM (16 heads x 8 groups are 128 blocks for 148 SMs); two (which share WQ, K1 and K2) where the
// heads are more. 2,048 tokens of 16 heads of 128 x 128 take 98 us here and 118 us in the kernel in front (B200), where the
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

// 16 and 4 bytes into shared memory, asynchronously
__device__ __forceinline__ void copy_16(float* smem, const float* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_4(float* smem, const float* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}

// ---- 32-bit products on the tensor cores ----------------------------------------------------------
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

// a b of eight channels or tokens, b given in its parts: the sum of the three products, in the tensor cores
__device__ __forceinline__ void piece_of(float (&d)[4], const uint32_t (&hi)[4], const uint32_t (&lo)[4], uint32_t bh0, uint32_t bh1, uint32_t bl0,
                                         uint32_t bl1) {
  mma_1688_first(d, lo, bh0, bh1);
  mma_1688(d, hi, bl0, bl1);
  mma_1688(d, hi, bh0, bh1);
}

// ---- what the kernels in front of the walk share ----------------------------------------------------
// A chunk's small matrices are lower triangular, [token i][token j], and are made and used in blocks of 8 x 8 tokens. Those below the
// diagonal are sums over channels of products of a row of token i, decayed on from its block's start, and a row of token j, decayed on to its
// block's end (and through the blocks between): no factor is above one, so nothing overflows and what underflows is nothing. They
// come off the tensor cores in the layout in which the substitution's products read them as their second operand, and are kept there
// split in two. Those on the diagonal are sums of running products, token by token, and are used so: a number that is not
// finite at token j must not meet the zeros of the tokens in front of it.
constexpr int NB = C / 8, BELOW = NB * (NB - 1) / 2;      // blocks; those below the diagonal
__host__ __device__ constexpr int below(int bi, int bj) { return bi * (bi - 1) / 2 + bj; }
struct Lower {
  float4 off[BELOW][32];               // a lane's two numbers (token i = lane / 4, tokens j = 2 (lane % 4) and the next): high parts, low parts
  float on[NB][64];                    // [token j][token i]
};
__device__ __forceinline__ float4 split_pair(float a, float b) {
  uint32_t ah, al, bh, bl;
  split(a, ah, al), split(b, bh, bl);
  return make_float4(__uint_as_float(ah), __uint_as_float(bh), __uint_as_float(al), __uint_as_float(bl));
}

// A decay exp(x) as it lies in shared memory: from a half to one as what it lacks of one, exp(x) - 1 (not above zero; the exponential's series
// up to x^10), else itself (above zero: one denormal is added). A decay next to one, as a number of its own, has few bits of what it takes
// away, and over the thousands of tokens that it keeps that was most of the error: read-outs of 2,048 tokens with decays around 0.9997 were
// 2.9e-6 off 64 bits, now 0.2e-6. It costs the gated rule's factors 3%.
__device__ __forceinline__ float kept_decay(float x) {
  float q = 1.f / 3628800.f;
  q = fmaf(q, x, 1.f / 362880.f), q = fmaf(q, x, 1.f / 40320.f), q = fmaf(q, x, 1.f / 5040.f), q = fmaf(q, x, 1.f / 720.f);
  q = fmaf(q, x, 1.f / 120.f), q = fmaf(q, x, 1.f / 24.f), q = fmaf(q, x, 1.f / 6.f), q = fmaf(q, x, 0.5f);
  return x < -0.6931472f || x > 0.f ? expf(x) + 1.4e-45f : fmaf(x * x, q, x);
}
__device__ __forceinline__ float rounded_decay(float kept) { return kept > 0.f ? kept : 1.0f + kept; }      // (zero is one denormal here)
__device__ __forceinline__ float2 whole_decay(float kept) {                                                // in two numbers
  const float one = 1.0f + kept;
  return kept > 0.f ? make_float2(kept - 1.4e-45f, 0.f) : make_float2(one, kept - (one - 1.0f));
}

// 1 / sqrt(x) in two numbers, the second from what the first's square lacks (zero for an x whose root's square would be subnormal). A row's
// length is an error of the whole row: in one number read-outs were up to 1.05 times as far from 64 bits as with pair sums in 32-bit
// multiply-adds throughout, in two they are 0.87 to 1.0 times as far.
__device__ __forceinline__ float2 one_over_root(float x) {
  const float y = 1.0f / sqrtf(x), p = y * y;
  return make_float2(y, x < 1e30f ? 0.5f * y * fmaf(-fmaf(y, y, -p), x, fmaf(-p, x, 1.0f)) : 0.f);
}

// A running product of decays in two numbers, so that it is rounded once however long it is: a head's one decay for all channels makes
// its rounding the whole row's (with single numbers the gated rule's read-outs were up to 1.1 times as far from 64 bits).
struct Product {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void by(float2 g) {
    const float p = hi * g.x;
    lo = fmaf(hi, g.y, fmaf(lo, g.x, fmaf(hi, g.x, -p))), hi = p;
  }
  __device__ __forceinline__ float of(float x) const { return fmaf(x, hi, x * lo); }
  __device__ __forceinline__ float2 both() const { return make_float2(hi, lo); }
  __device__ __forceinline__ float value() const { return hi + lo; }
};

// The block (bi, bj) below the diagonal of two matrices at once: rows 0 to 7 of the product's 16 belong to `first`, the others to
// `second` [tokens of bi][LD], the second operand is `with` [tokens of bj][LD]; through [NB][DIM]: whole blocks' decays.
template <int DIM, int LD>
__device__ __forceinline__ void block_below(float (&acc)[4], const float* first, const float* second, const float* with, const float2* through, int bi,
                                            int bj, int lane) {
  const int at = (lane >> 2) * LD + 2 * (lane & 3);
  const float *a = first + bi * 8 * LD + at, *b = second + bi * 8 * LD + at, *c = with + bj * 8 * LD + at;
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] = 0.f;
#pragma unroll 1
  for (int s0 = 0; s0 < DIM; s0 += 32) {
    float sum[2][4];                     // the pieces two by two, so that fewer of the additions are of the whole sum
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int s = s0 + 8 * i;
      const float2 x = *reinterpret_cast<const float2*>(a + s), y = *reinterpret_cast<const float2*>(b + s);
      float2 z = *reinterpret_cast<const float2*>(c + s);
      for (int between = bj + 1; between < bi; ++between) {
        const float4 g = *reinterpret_cast<const float4*>(through + between * DIM + s + 2 * (lane & 3));
        z.x = fmaf(z.x, g.x, z.x * g.y), z.y = fmaf(z.y, g.z, z.y * g.w);
      }
      uint32_t hi[4], lo[4], h0, l0, h1, l1;
      split(x.x, hi[0], lo[0]), split(y.x, hi[1], lo[1]), split(x.y, hi[2], lo[2]), split(y.y, hi[3], lo[3]);
      split(z.x, h0, l0), split(z.y, h1, l1);
      float piece[4];
      piece_of(piece, hi, lo, h0, h1, l0, l1);
#pragma unroll
      for (int e = 0; e < 4; ++e) sum[i >> 1][e] = i & 1 ? sum[i >> 1][e] + piece[e] : piece[e];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] += sum[0][e] + sum[1][e];
  }
}

// The substitution, a warp per 16 columns in the accumulators' layout: [e] is column lane / 4 + 8 (e / 2), token 2 (lane % 4) + (e & 1) of
// a block. take holds what the tokens in front take off (or, for a second matrix, add to) a row, summed by itself: it is small beside
// the row, and what is added last is rounded last. This: the block's own tokens, one after another. now(e): token e & 1's number as it stands;
// where a lane's token is behind token j it loses m1_ij times it, and from j on `more` gains m2_ij times it.
template <class Now>
__device__ __forceinline__ void on_diagonal(const float* m1, const float* m2, int lane, float (&take)[4], float (&more)[4], Now&& now) {
  const int tig = lane & 3;
  const float *a = m1 + 2 * tig, *b = m2 + 2 * tig;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 x = *reinterpret_cast<const float2*>(a + j * 8), z = *reinterpret_cast<const float2*>(b + j * 8);
    const float y0 = __shfl_sync(0xffffffffu, now(j & 1), (lane & 28) | (j >> 1));
    const float y1 = __shfl_sync(0xffffffffu, now(2 + (j & 1)), (lane & 28) | (j >> 1));
    if (2 * tig > j) take[0] = fmaf(-x.x, y0, take[0]), take[2] = fmaf(-x.x, y1, take[2]);
    if (2 * tig + 1 > j) take[1] = fmaf(-x.y, y0, take[1]), take[3] = fmaf(-x.y, y1, take[3]);
    if (2 * tig >= j) more[0] = fmaf(z.x, y0, more[0]), more[2] = fmaf(z.x, y1, more[2]);
    if (2 * tig + 1 >= j) more[1] = fmaf(z.y, y0, more[1]), more[3] = fmaf(z.y, y1, more[3]);
  }
}
// The later blocks' share of a finished block bj: y its numbers.
__device__ __forceinline__ void below_diagonal(const Lower& m1, const Lower& m2, int bj, int lane, const float (&y)[4], float (&take)[NB][4],
                                               float (&more)[NB][4]) {
  uint32_t hi[4], lo[4];
  split(y[0], hi[0], lo[0]), split(y[2], hi[1], lo[1]), split(y[1], hi[2], lo[2]), split(y[3], hi[3], lo[3]);
#pragma unroll
  for (int bi = 1; bi < NB; ++bi) {
    if (bi <= bj) continue;
    const float4 f = m1.off[below(bi, bj)][lane], k = m2.off[below(bi, bj)][lane];
    float p[4], q[4];
    piece_of(p, hi, lo, __float_as_uint(f.x), __float_as_uint(f.y), __float_as_uint(f.z), __float_as_uint(f.w));
    piece_of(q, hi, lo, __float_as_uint(k.x), __float_as_uint(k.y), __float_as_uint(k.z), __float_as_uint(k.w));
#pragma unroll
    for (int e = 0; e < 4; ++e) take[bi][e] -= p[e], more[bi][e] += q[e];
  }
}
// A block's numbers into rows row0 .. of W or Q, or into columns of tokens from 8 bi on (VP, OP, V).
__device__ __forceinline__ void store_tile_rows(float* block, const Layout& lay, int row0, int col0, int lane, const float (&x)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) block[lay.wq(row0 + 2 * (lane & 3) + (e & 1), col0 + (lane >> 2) + 8 * (e >> 1))] = x[e];
}
__device__ __forceinline__ void store_tile_columns(float* to, int col0, int bi, int lane, const float (&x)[4]) {
  float* p = to + (col0 + (lane >> 2)) * C + bi * 8 + 2 * (lane & 3);
  *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  *reinterpret_cast<float2*>(p + 8 * C) = make_float2(x[2], x[3]);
}

// ---- the walk ------------------------------------------------------------------------------------
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
