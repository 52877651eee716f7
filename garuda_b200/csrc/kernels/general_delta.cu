// The generalized delta rule: a recurrent mixer whose state per request and head is a matrix
// S [dim, vdim] in 32-bit. Per token, with r, k, v the projected rows, w a decay and a a removal
// rate per head and key channel, and u = k / sqrt(sum k^2 + 1e-6) the head's unit key:
//     S <- diag(w) S - (a * u) (u^T S) + k v^T      (both terms read the old S)
//     o  = S^T r
//     w  = exp(-c sigmoid(z + w0)),   a = sigmoid(y + a0)
// with z the decay's pre-activation (a low-rank pair of products), y the removal's, c a constant.
//
// Column c of S, u^T S at c and o_c involve no other column, so a request's tokens are walked in
// order with no exchange between columns. Kernels, all 32-bit arithmetic:
//   gdelta_prepare      a block per token: decays, removal rates, unit keys
//   gdelta_recurrence   eight threads share a column (every eighth row each, in registers) and
//                       exchange two sums per token by shuffles; a token's r, u, w, a*u, k come
//                       through shared memory, eight (or four) tokens at a time in two buffers
//   gdelta_decode       all of it, with the read-out's norm, weight and gate, for steps of one
//                       token per request: a block per (request, head)
//   gdelta_chunk_factors, delta_chunk::walk
//                       the same for long stretches of tokens in a bfloat16 run, 32 tokens at a time
//                       (delta_chunk.cuh)
// The read-out's norm for longer steps is delta_out (delta_rule.cu). In the token-by-token kernels a token's
// result depends on its request's earlier tokens only through the state, which is carried bit for bit; the
// chunked ones add the same terms in another order, so there a cut moves the last bits.
#include <type_traits>

#include "common.cuh"
#include "delta_chunk.cuh"

namespace {

__device__ __forceinline__ float sigmoid(float z) { return gb::over(1.0f + expf(-z)); }

// proj [T, P]: columns r | k | v | removal logits | ...; each block H dim wide (v: H vdim).
// zdec [T, PZ]: the decay's pre-activation, H dim wide.
// prep [T, W]: r | u | w | a*u | k  (H dim each) | v (H vdim).
__global__ void __launch_bounds__(256)
gdelta_prepare_kernel(const float* __restrict__ proj, int P, int col_r, int col_k, int col_v, int col_a,
                      const float* __restrict__ zdec, int PZ, const float* __restrict__ w0, const float* __restrict__ a0,
                      float decay_scale, float* __restrict__ prep, int W, int H, int dim, int vdim,
                      const int32_t* __restrict__ token_req, const int32_t* __restrict__ cu_q, int below) {
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  const size_t t = blockIdx.x;
  if (below > 0 && cu_q[token_req[t] + 1] - cu_q[token_req[t]] >= below) return;      // the chunked kernels' request
  const float* row = proj + t * P;
  float* out = prep + t * W;
  const int HD = H * dim;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int h = warp; h < H; h += warps) {
    const float* k = row + col_k + h * dim;
    float ss = 0.f;
    for (int d = lane; d < dim; d += 32) ss = fmaf(k[d], k[d], ss);
    const float inv = 1.0f / sqrtf(gb::warp_sum(ss) + 1e-6f);
    for (int d = lane; d < dim; d += 32) {
      const int c = h * dim + d;
      const float u = k[d] * inv;
      out[c] = row[col_r + c];
      out[HD + c] = u;
      out[2 * HD + c] = expf(-decay_scale * sigmoid(zdec[t * PZ + c] + w0[c]));
      out[3 * HD + c] = sigmoid(row[col_a + c] + a0[c]) * u;
      out[4 * HD + c] = k[d];
    }
  }
  for (int c = threadIdx.x; c < H * vdim; c += blockDim.x) out[5 * HD + c] = row[col_v + c];
}

constexpr int SPLIT = 8;        // threads that share a column of S: thread `sub` holds the rows d with d % 8 == sub
constexpr int REC_THREADS = 128, REC_COLS = REC_THREADS / SPLIT;
constexpr int VECS = 5;         // r, u, w, a*u, k

// grid (H, R, ceil(vdim / 16)), 128 threads: 16 columns of S, eight threads a column. Each of the
// eight sums its rows in ascending order and the eight are added as a tree, ((0 + 1) + (2 + 3)) +
// ((4 + 5) + (6 + 7)): the same sums, in the same order, as the eight interleaved partial sums of
// the one-token kernel below. EXACT: dim == MAXD, no row of a thread is beyond the head's.
template <int MAXD, bool EXACT, int CHUNK>
__global__ void __launch_bounds__(REC_THREADS)
gdelta_recurrence_kernel(const float* __restrict__ prep, int W, const int32_t* __restrict__ cu_q,
                         const int32_t* __restrict__ slots, float* __restrict__ state, long long state_stride, int H,
                         int dim, int vdim, int below, float* __restrict__ out) {
  gb::pdl_wait();
  if (below > 0 && cu_q[blockIdx.y + 1] - cu_q[blockIdx.y] >= below) return;      // the chunked kernels' request
  constexpr int MINE = MAXD / SPLIT;
  extern __shared__ __align__(16) float stage[];      // 2 x [CHUNK][VECS SPLIT per + 16 + 4]
  const int per = ((dim + SPLIT - 1) / SPLIT + 3) / 4 * 4 + 4;
  const int tok_floats = VECS * SPLIT * per + REC_COLS + 4;
  const int h = blockIdx.x, r = blockIdx.y;
  const int sub = threadIdx.x % SPLIT;
  const int col0 = blockIdx.z * REC_COLS, mycol = threadIdx.x / SPLIT, col = col0 + mycol;
  const bool active = col < vdim;
  const int slot = slots[r];
  const int t0 = cu_q[r], t1 = cu_q[r + 1];
  const int HD = H * dim;
  const int off_v = VECS * HD + h * vdim + col0;
  const int ncols = min(REC_COLS, vdim - col0);
  float* S_g = (slot >= 0 && active) ? state + (size_t)slot * state_stride + (size_t)h * dim * vdim + col : nullptr;
  float S[MINE];
#pragma unroll
  for (int i = 0; i < MINE; ++i) {
    const int d = i * SPLIT + sub;
    S[i] = (d < dim && S_g != nullptr) ? S_g[(size_t)d * vdim] : 0.f;
  }
  auto fetch = [&](int c0, int buf) {
    const int n = min(CHUNK, t1 - c0);
    float* dst = stage + (size_t)buf * CHUNK * tok_floats;
    for (int i = threadIdx.x; i < n * dim; i += REC_THREADS) {
      const int tt = i / dim, d = i % dim;
      const float* row = prep + (size_t)(c0 + tt) * W + h * dim + d;
      float* to = dst + tt * tok_floats + (d % SPLIT) * per + d / SPLIT;
#pragma unroll
      for (int v = 0; v < VECS; ++v) delta_chunk::copy_4(to + v * SPLIT * per, row + v * HD);
    }
    for (int i = threadIdx.x; i < n * ncols; i += REC_THREADS) {
      const int tt = i / ncols, c = i % ncols;
      delta_chunk::copy_4(dst + tt * tok_floats + VECS * SPLIT * per + c, prep + (size_t)(c0 + tt) * W + off_v + c);
    }
  };
  if (t0 < t1) fetch(t0, 0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  int buf = 0;
  for (int c0 = t0; c0 < t1; c0 += CHUNK, buf ^= 1) {
    const int n = min(CHUNK, t1 - c0);
    if (c0 + CHUNK < t1) fetch(c0 + CHUNK, buf ^ 1);       // that buffer was read two rounds ago, behind a barrier
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float* cur = stage + (size_t)buf * CHUNK * tok_floats;
    // unrolled: a token's read-out (its sum and shuffles) is off the path to the next token's state and overlaps it
#pragma unroll 4
    for (int tt = 0; tt < n; ++tt) {
      const float* tok = cur + tt * tok_floats;
      const float* sr = tok + sub * per;
      const float* su = sr + SPLIT * per;
      const float* sw = su + SPLIT * per;
      const float* sa = sw + SPLIT * per;
      const float* sk = sa + SPLIT * per;
      const float v = active ? tok[VECS * SPLIT * per + mycol] : 0.f;
      float acc = 0.f;
#pragma unroll
      for (int i4 = 0; i4 < MINE; i4 += 4) {
        if (!EXACT && i4 * SPLIT >= dim) break;         // pieces beyond the head's rows are not in shared memory
        const float4 u4 = *reinterpret_cast<const float4*>(su + i4);
        const float uu[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (EXACT || (i4 + j) * SPLIT + sub < dim) acc = fmaf(S[i4 + j], uu[j], acc);
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 4);
      float o = 0.f;
#pragma unroll
      for (int i4 = 0; i4 < MINE; i4 += 4) {
        if (!EXACT && i4 * SPLIT >= dim) break;
        const float4 w4 = *reinterpret_cast<const float4*>(sw + i4);
        const float4 a4 = *reinterpret_cast<const float4*>(sa + i4);
        const float4 k4 = *reinterpret_cast<const float4*>(sk + i4);
        const float4 r4 = *reinterpret_cast<const float4*>(sr + i4);
        const float ww[4] = {w4.x, w4.y, w4.z, w4.w}, aa[4] = {a4.x, a4.y, a4.z, a4.w};
        const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (EXACT || (i4 + j) * SPLIT + sub < dim) {
            S[i4 + j] = fmaf(kk[j], v, fmaf(-aa[j], acc, ww[j] * S[i4 + j]));
            o = fmaf(S[i4 + j], rr[j], o);
          }
      }
      o += __shfl_xor_sync(0xffffffffu, o, 1);
      o += __shfl_xor_sync(0xffffffffu, o, 2);
      o += __shfl_xor_sync(0xffffffffu, o, 4);
      if (active && sub == 0) out[(size_t)(c0 + tt) * H * vdim + h * vdim + col] = o;
    }
    __syncthreads();
  }
  // only now may the next kernel in the stream start: its blocks would wait beside these for the whole walk
  gb::pdl_launch_dependents();
  if (S_g != nullptr) {
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      const int d = i * SPLIT + sub;
      if (d < dim) S_g[(size_t)d * vdim] = S[i];
    }
  }
}

// What the walk of delta_chunk.cuh needs of a chunk and a head. With D_i the product of the decays up to token i and
// alpha = a * u, the row x_i = u_i^T S of token i, taken from the state in front of it, is
//     x_i = (D_i-1 u_i)^T S_0 + sum_{j<i} F_ij v_j - E_ij x_j,   E_ij = sum_d u_i alpha_j D_i-1 / D_j,   F_ij likewise with k_j
//     o_i = (D_i r_i)^T S_0 + sum_{j<=i} H_ij v_j - G_ij x_j,    G_ij = sum_d r_i alpha_j D_i / D_j,     H_ij likewise with k_j
// so  W = (I + E)^-1 (D u),   VP = -(I + E)^-1 F v,   Q = D r - G W,   OP = H v + G VP,   K1_j = alpha_j D_last / D_j,   K2_j = k_j
// D_last / D_j, and the walk's Y is -x. As for the gated rule (delta_rule.cu), in blocks of 8 tokens: on the tensor cores off the
// diagonal, in 32-bit multiply-adds on it. Bound as that kernel is. With running products for all pairs, a thread per column in the
// substitution and rows fetched by the warps that use them 170 us for 2,048 tokens of 32 heads of 64 x 64, now 115.
// grid (numbers, H), 256 threads.
template <int DIM>
struct FactorsSmem {
  delta_chunk::Lower E, F, G, H;
  // [tokens][DIM + 8] each: u and r, then decayed on from their block's start (u up to the token in front of it); alpha and k, then decayed on
  // to their block's end; decays (kept_decay)
  float u[delta_chunk::C * (DIM + 8)], r[delta_chunk::C * (DIM + 8)], a[delta_chunk::C * (DIM + 8)], k[delta_chunk::C * (DIM + 8)],
      w[delta_chunk::C * (DIM + 8)];
  float2 through[delta_chunk::NB * DIM];         // whole blocks' decays (delta_chunk::Product)
};

template <int DIM>
__global__ void __launch_bounds__(256, DIM == 64 ? 3 : 2)
gdelta_chunk_factors_kernel(const float* __restrict__ proj, int P, int col_r, int col_k, int col_v, int col_a,
                            const float* __restrict__ zdec, int PZ, const float* __restrict__ w0, const float* __restrict__ a0,
                            float decay_scale, const int32_t* __restrict__ cu_q, float* __restrict__ blocks, int R, int H, int vdim,
                            int cut) {
  using namespace delta_chunk;
  using delta_chunk::C;
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  constexpr int LD = DIM + 8, VEC = DIM / 32;
  extern __shared__ __align__(16) unsigned char raw[];
  FactorsSmem<DIM>& sm = *reinterpret_cast<FactorsSmem<DIM>*>(raw);
  float *su = sm.u, *sr = sm.r, *sa = sm.a, *sk = sm.k, *sw = sm.w;
  const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int r, first, n, at;
  if (!find_chunk(blockIdx.x, cu_q, R, cut, r, first, n, at)) return;
  const Layout lay{DIM, vdim, 1};
  float* block = blocks + ((size_t)blockIdx.x * H + h) * lay.floats();
  const float* row0 = proj + (size_t)first * P;
  auto rows = [&](float* to, const float* from, int pitch) {      // all at once; 16 bytes a copy where rows start on 16 bytes
    if (pitch % 4 == 0 && ((uintptr_t)from & 15) == 0) {
      for (int i = tid; i < n * (DIM / 4); i += 256)
        copy_16(to + i / (DIM / 4) * LD + i % (DIM / 4) * 4, from + (size_t)(i / (DIM / 4)) * pitch + i % (DIM / 4) * 4);
    } else {
      for (int i = tid; i < n * DIM; i += 256) copy_4(to + i / DIM * LD + i % DIM, from + (size_t)(i / DIM) * pitch + i % DIM);
    }
  };
  rows(sk, row0 + col_k + h * DIM, P);
  rows(sa, row0 + col_a + h * DIM, P);
  rows(sw, zdec + (size_t)first * PZ + h * DIM, PZ);
  rows(sr, row0 + col_r + h * DIM, P);
  asm volatile("cp.async.commit_group;" ::: "memory");
  float rate[VEC], decay[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) rate[e] = a0[h * DIM + lane + 32 * e], decay[e] = w0[h * DIM + lane + 32 * e];
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int t = warp; t < C; t += 8) {
    float k[VEC], ss = 0.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e) k[e] = t < n ? sk[t * LD + lane + 32 * e] : 0.f, ss = fmaf(k[e], k[e], ss);
    const float inv = 1.0f / sqrtf(gb::warp_sum(ss) + 1e-6f);
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const int d = t * LD + lane + 32 * e;
      const float u = k[e] * inv;
      su[d] = u;
      sa[d] = t < n ? sigmoid(sa[d] + rate[e]) * u : 0.f;
      sw[d] = t < n ? kept_decay(-decay_scale * sigmoid(sw[d] + decay[e])) : 0.f;
      if (t >= n) sk[d] = sr[d] = 0.f;
    }
  }
  __syncthreads();
  {
    // the matrices on the diagonal: a warp has four keys j, decayed on from token to token up to their block's end
    const int j0 = warp * 4, j1 = (warp | 1) * 4 + 4, d0 = lane * VEC;
    pair_t pa[4][VEC / 2], pk[4][VEC / 2];                // alpha_j and k_j
    auto row = [&](const float* m, int i, pair_t (&x)[VEC / 2]) {
      if (VEC == 4) {
        const pair2_t f = *reinterpret_cast<const pair2_t*>(m + i * LD + d0);
        x[0] = f.a, x[VEC / 2 - 1] = f.b;
      } else {
        x[0] = *reinterpret_cast<const pair_t*>(m + i * LD + d0);
      }
    };
    auto decays = [&](int i, pair_t (&x)[VEC / 2]) {
      row(sw, i, x);
#pragma unroll
      for (int e = 0; e < VEC / 2; ++e) x[e] = make_pair(rounded_decay(both(x[e]).x), rounded_decay(both(x[e]).y));
    };
    auto dot = [](const pair_t (&a)[VEC / 2], const pair_t (&b)[VEC / 2]) {
      pair_t s = mul2(a[0], b[0]);
#pragma unroll
      for (int e = 1; e < VEC / 2; ++e) s = fma2(a[e], b[e], s);
      const float2 f = both(s);
      return f.x + f.y;
    };
    auto keep = [&](int i, float (&before)[8], float (&after)[8]) {
      const float b = sum_of_eight(before, lane), a = sum_of_eight(after, lane);
      const int which = lane >> 2, j = j0 + (which & 3), place = (j & 7) * 8 + (i & 7);
      if ((lane & 3) == 0 && j <= i) {
        if (j < i) (which < 4 ? sm.E : sm.F).on[j >> 3][place] = b;
        (which < 4 ? sm.G : sm.H).on[j >> 3][place] = a;
      }
    };
#pragma unroll
    for (int ii = 0; ii < 4; ++ii) {       // the tokens of the four keys themselves
      const int i = j0 + ii;
      pair_t w[VEC / 2], u[VEC / 2], x[VEC / 2];
      decays(i, w), row(su, i, u), row(sr, i, x);
      row(sa, i, pa[ii]), row(sk, i, pk[ii]);
      float before[8], after[8];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        before[jj] = jj < ii ? dot(pa[jj], u) : 0.f, before[4 + jj] = jj < ii ? dot(pk[jj], u) : 0.f;
        if (jj < ii) {
#pragma unroll
          for (int e = 0; e < VEC / 2; ++e) pa[jj][e] = mul2(pa[jj][e], w[e]), pk[jj][e] = mul2(pk[jj][e], w[e]);
        }
        after[jj] = jj <= ii ? dot(pa[jj], x) : 0.f, after[4 + jj] = jj <= ii ? dot(pk[jj], x) : 0.f;
      }
      keep(i, before, after);
    }
    for (int i = j0 + 4; i < j1; ++i) {
      pair_t w[VEC / 2], u[VEC / 2], x[VEC / 2];
      decays(i, w), row(su, i, u), row(sr, i, x);
      float before[8], after[8];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        before[jj] = dot(pa[jj], u), before[4 + jj] = dot(pk[jj], u);
#pragma unroll
        for (int e = 0; e < VEC / 2; ++e) pa[jj][e] = mul2(pa[jj][e], w[e]), pk[jj][e] = mul2(pk[jj][e], w[e]);
        after[jj] = dot(pa[jj], x), after[4 + jj] = dot(pk[jj], x);
      }
      keep(i, before, after);
    }
  }
  __syncthreads();
  // decayed on within a block of tokens
  for (int i = tid; i < NB * DIM; i += 256) {
    const int c = i % DIM, at0 = i / DIM * 8 * LD + c;
    float w[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) w[t] = sw[at0 + t * LD];
    Product on, behind;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      su[at0 + t * LD] = on.of(su[at0 + t * LD]);
      on.by(whole_decay(w[t]));
      sr[at0 + t * LD] = on.of(sr[at0 + t * LD]);
    }
    sm.through[i] = on.both();
#pragma unroll
    for (int t = 7; t >= 0; --t) {
      sa[at0 + t * LD] = behind.of(sa[at0 + t * LD]), sk[at0 + t * LD] = behind.of(sk[at0 + t * LD]);
      behind.by(whole_decay(w[t]));
    }
  }
  __syncthreads();
  for (int task = warp; task < 2 * BELOW; task += 8) {
    const int which = task >> 1, bi = which < 1 ? 1 : which < 3 ? 2 : 3, bj = which - below(bi, 0);
    float acc[4];
    block_below<DIM, LD>(acc, su, sr, task & 1 ? sk : sa, sm.through, bi, bj, lane);
    (task & 1 ? sm.F : sm.E).off[which][lane] = split_pair(acc[0], acc[1]);
    (task & 1 ? sm.H : sm.G).off[which][lane] = split_pair(acc[2], acc[3]);
  }
  for (int i = tid; i < NB * DIM; i += 256) {              // K1, K2 and the chunk's whole decay
    const int c = i % DIM, bj = i / DIM;
    Product behind;
    float x[8], y[8];
#pragma unroll
    for (int b = NB - 1; b > 0; --b)
      if (b > bj) behind.by(sm.through[b * DIM + c]);
#pragma unroll
    for (int t = 0; t < 8; ++t) x[t] = behind.of(sa[(bj * 8 + t) * LD + c]), y[t] = behind.of(sk[(bj * 8 + t) * LD + c]);
    float4* to = reinterpret_cast<float4*>(block + lay.k1(bj * 8, c));
    to[0] = make_float4(x[0], x[1], x[2], x[3]), to[1] = make_float4(x[4], x[5], x[6], x[7]);
    to = reinterpret_cast<float4*>(block + lay.k1(C + bj * 8, c));
    to[0] = make_float4(y[0], y[1], y[2], y[3]), to[1] = make_float4(y[4], y[5], y[6], y[7]);
    if (bj == 0) {
      behind.by(sm.through[c]);
      block[lay.last() + c] = behind.value();
    }
  }
  __syncthreads();
  const int g = lane >> 2, tig = lane & 3;
  for (int col0 = warp * 16; col0 < DIM + vdim; col0 += 128) {
    float take[NB][4], more[NB][4];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int e = 0; e < 4; ++e) take[b][e] = more[b][e] = 0.f;
    if (col0 < DIM) {                    // D u, and what D r loses
      Product front[2];       // the blocks in front
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float x[4], y[4], q[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = front[e >> 1].of(su[(b * 8 + 2 * tig + (e & 1)) * LD + col0 + g + 8 * (e >> 1)]);
        on_diagonal(sm.E.on[b], sm.G.on[b], lane, take[b], more[b], [&](int e) { return x[e] + take[b][e]; });
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          y[e] = x[e] + take[b][e];
          q[e] = front[e >> 1].of(sr[(b * 8 + 2 * tig + (e & 1)) * LD + col0 + g + 8 * (e >> 1)]) - more[b][e];
        }
        store_tile_rows(block, lay, b * 8, col0, lane, y);
        store_tile_rows(block, lay, C + b * 8, col0, lane, q);
        if (b + 1 < NB) below_diagonal(sm.E, sm.G, b, lane, y, take, more);
        front[0].by(sm.through[b * DIM + col0 + g]), front[1].by(sm.through[b * DIM + col0 + g + 8]);
      }
    } else {                             // -F v, then VP; H v and what it gains
      const int v0 = col0 - DIM;
      const float* from = row0 + col_v + h * vdim + v0 + g;
      float v[NB][4];
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = b * 8 + 2 * tig + (e & 1);
          v[b][e] = t < n ? from[(size_t)t * P + 8 * (e >> 1)] : 0.f;
        }
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        store_tile_columns(block + lay.v(), v0, b, lane, v[b]);
        on_diagonal(sm.F.on[b], sm.H.on[b], lane, take[b], more[b], [&](int e) { return v[b][e]; });
        on_diagonal(sm.E.on[b], sm.G.on[b], lane, take[b], more[b], [&](int e) { return take[b][e]; });
        store_tile_columns(block + lay.vp(), v0, b, lane, take[b]);
        store_tile_columns(block + lay.op(), v0, b, lane, more[b]);
        if (b + 1 < NB) {
          below_diagonal(sm.F, sm.H, b, lane, v[b], take, more);
          below_diagonal(sm.E, sm.G, b, lane, take[b], take, more);
        }
      }
    }
  }
}

// A step of one token per request: grid (H, R), vdim threads (a column of S each, rounded up to a
// warp). The state column lives in registers for the one token: read, updated, written. The sums
// are taken as the kernel for longer steps takes them, so a token's result is the same bits
// whichever kernel ran it.
template <int MAXD, typename OT>
__global__ void __launch_bounds__(256)
gdelta_decode_kernel(const float* __restrict__ proj, int P, int col_r, int col_k, int col_v, int col_a, int col_g,
                     const float* __restrict__ zdec, int PZ, const float* __restrict__ w0, const float* __restrict__ a0,
                     float decay_scale, const float* __restrict__ norm_w, float eps, const int32_t* __restrict__ slots,
                     float* __restrict__ state, long long state_stride, int H, int dim, int vdim, OT* __restrict__ out) {
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  extern __shared__ float sm[];          // r, u, w, a*u, k [dim each], o [vdim]
  float* sr = sm;
  float* su = sm + dim;
  float* sw = sm + 2 * dim;
  float* sa = sm + 3 * dim;
  float* sk = sm + 4 * dim;
  float* so = sm + 5 * dim;
  const int h = blockIdx.x;
  const size_t t = blockIdx.y;            // one token per request: row t is request t
  const int slot = slots[t];
  const float* row = proj + t * P;
  const int lane = threadIdx.x & 31;
  // the unit key: every warp takes the sum itself (a lane's channels in ascending order, then the tree)
  float ss = 0.f;
  for (int d = lane; d < dim; d += 32) {
    const float k = row[col_k + h * dim + d];
    ss = fmaf(k, k, ss);
  }
  const float inv = 1.0f / sqrtf(gb::warp_sum(ss) + 1e-6f);
  for (int d = threadIdx.x; d < dim; d += blockDim.x) {
    const int c = h * dim + d;
    const float k = row[col_k + c], u = k * inv;
    sr[d] = row[col_r + c];
    su[d] = u;
    sw[d] = expf(-decay_scale * sigmoid(zdec[t * PZ + c] + w0[c]));
    sa[d] = sigmoid(row[col_a + c] + a0[c]) * u;
    sk[d] = k;
  }
  __syncthreads();
  const int col = threadIdx.x;
  const bool active = col < vdim;
  float o_val = 0.f;
  if (active) {
    const float v = row[col_v + h * vdim + col];
    float* S_g = slot >= 0 ? state + (size_t)slot * state_stride + (size_t)h * dim * vdim + col : nullptr;
    float S[MAXD];
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
      if (d < dim) {
        S[d] = S_g != nullptr ? S_g[(size_t)d * vdim] : 0.f;
        acc[d & 7] = fmaf(S[d], su[d], acc[d & 7]);
      }
    const float dot = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
    float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
      if (d < dim) {
        S[d] = fmaf(sk[d], v, fmaf(-sa[d], dot, sw[d] * S[d]));
        o[d & 7] = fmaf(S[d], sr[d], o[d & 7]);
        if (S_g != nullptr) S_g[(size_t)d * vdim] = S[d];
      }
    o_val = ((o[0] + o[1]) + (o[2] + o[3])) + ((o[4] + o[5]) + (o[6] + o[7]));
    so[col] = o_val;
  }
  __syncthreads();
  float sq = 0.f;
  for (int c = lane; c < vdim; c += 32) sq = fmaf(so[c], so[c], sq);
  const float scale = 1.0f / sqrtf(gb::warp_sum(sq) / (float)vdim + eps);
  if (active) {
    const float gate = row[col_g + h * vdim + col];
    out[(t * H + h) * vdim + col] = gb::from_float<OT>((o_val * scale) * norm_w[h * vdim + col] * sigmoid(gate));
  }
}

template <typename F>
int by_dim(int dim, const char* what, F&& f) {
  if (dim <= 32) return f(std::integral_constant<int, 32>());
  if (dim <= 64) return f(std::integral_constant<int, 64>());
  if (dim <= 128) return f(std::integral_constant<int, 128>());
  if (dim <= 256) return f(std::integral_constant<int, 256>());
  return gb::fail(GB_UNSUPPORTED, "%s: %d key channels per head (at most 256)", what, dim);
}

}  // namespace

// below (here and in gdelta_recurrence): only requests with fewer tokens in the step than this (0: all).
GB_EXPORT int gb_gdelta_prepare(const float* proj, int P, int col_r, int col_k, int col_v, int col_a, const float* zdec,
                                int PZ, const float* w0, const float* a0, float decay_scale, float* prep, int W, int T, int H,
                                int dim, int vdim, const int32_t* token_req, const int32_t* cu_q, int below, cudaStream_t stream) {
  if (T <= 0) return GB_OK;
  if (H < 1 || dim < 1 || vdim < 1) return gb::fail(GB_BAD_ARGUMENT, "gdelta_prepare: sizes");
  if (W != 5 * H * dim + H * vdim || PZ < H * dim) return gb::fail(GB_BAD_ARGUMENT, "gdelta_prepare: row widths");
  return gb::check_pdl_launch(gb::launch_pdl(gdelta_prepare_kernel, dim3(T), dim3(256), 0, stream, dim3(1, 1, 1), proj, P, col_r,
                                             col_k, col_v, col_a, zdec, PZ, w0, a0, decay_scale, prep, W, H, dim, vdim, token_req, cu_q, below),
                              "gdelta_prepare");
}

GB_EXPORT int gb_gdelta_recurrence(const float* prep, int W, const int32_t* cu_q, const int32_t* slots, float* state,
                                   long long state_stride, int R, int H, int dim, int vdim, int below, float* out, cudaStream_t stream) {
  if (R <= 0) return GB_OK;
  if (H < 1 || dim < 1 || vdim < 1) return gb::fail(GB_BAD_ARGUMENT, "gdelta_recurrence: sizes");
  const dim3 grid(H, R, (vdim + REC_COLS - 1) / REC_COLS);
  const int per = ((dim + SPLIT - 1) / SPLIT + 3) / 4 * 4 + 4;
  const size_t tok = (size_t)(VECS * SPLIT * per + REC_COLS + 4) * sizeof(float);
  // eight tokens at a time where two buffers of them fit in 48 KB (up to 64 key channels), else four (47 KB at 256)
  const bool eight = 2 * 8 * tok <= 48 * 1024;
  const size_t smem = 2 * (eight ? 8 : 4) * tok;
  if (smem > 48 * 1024) return gb::fail(GB_UNSUPPORTED, "gdelta_recurrence: %d key channels per head", dim);
  return by_dim(dim, "gdelta_recurrence", [&](auto maxd) -> int {
    constexpr int MAXD = decltype(maxd)::value;
    auto kernel = eight ? (dim == MAXD ? gdelta_recurrence_kernel<MAXD, true, 8> : gdelta_recurrence_kernel<MAXD, false, 8>)
                        : (dim == MAXD ? gdelta_recurrence_kernel<MAXD, true, 4> : gdelta_recurrence_kernel<MAXD, false, 4>);
    return gb::check_pdl_launch(gb::launch_after(kernel, grid, dim3(REC_THREADS), smem, stream, dim3(1, 1, 1), prep, W, cu_q, slots,
                                               state, state_stride, H, dim, vdim, below, out),
                                "gdelta_recurrence");
  });
}

// Whether the chunked kernels take these sizes, and the floats of `blocks` for a step of T tokens, `walked` requests of which have at
// least `cut` (0: they do not).
GB_EXPORT long long gb_gdelta_chunk_floats(int T, int walked, int H, int dim, int vdim) {
  if (T <= 0 || walked <= 0 || H < 1 || H > 65535 || walked > 65535 || !delta_chunk::takes(dim, vdim)) return 0;
  return (long long)delta_chunk::chunk_numbers(T, walked) * H * delta_chunk::Layout{dim, vdim, 1}.floats();
}

// Requests of at least `cut` tokens: everything from the projected rows to the read-out o [T, H vdim] and the state. The rows
// are those of gdelta_prepare; walked: how many such requests the step has; blocks starts on 16 bytes.
GB_EXPORT int gb_gdelta_chunk(const float* proj, int P, int col_r, int col_k, int col_v, int col_a, const float* zdec, int PZ,
                              const float* w0, const float* a0, float decay_scale, const int32_t* cu_q, const int32_t* slots,
                              float* state, long long state_stride, float* blocks, int T, int R, int walked, int H, int dim, int vdim, int cut,
                              float* out, cudaStream_t stream) {
  if (T <= 0 || R <= 0 || walked <= 0) return GB_OK;
  if (R > 65535 || gb_gdelta_chunk_floats(T, walked, H, dim, vdim) == 0)
    return gb::fail(GB_UNSUPPORTED, "gdelta_chunk: %d heads of %d x %d", H, dim, vdim);
  if (PZ < H * dim) return gb::fail(GB_BAD_ARGUMENT, "gdelta_chunk: row widths");
  if ((uintptr_t)blocks & 15) return gb::fail(GB_BAD_ARGUMENT, "gdelta_chunk: blocks start on 16 bytes");
  const int numbers = delta_chunk::chunk_numbers(T, walked);
  const size_t smem = dim == 128 ? sizeof(FactorsSmem<128>) : sizeof(FactorsSmem<64>);
  auto kernel = dim == 128 ? gdelta_chunk_factors_kernel<128> : gdelta_chunk_factors_kernel<64>;
  static gb::OncePerDevice configured[2];
  if (configured[dim == 128].needed()) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "gdelta_chunk: %s", cudaGetErrorString(e));
    configured[dim == 128].done();
  }
  const int rc = gb::check_pdl_launch(
      gb::launch_pdl(kernel, dim3(numbers, H), dim3(256), smem, stream, dim3(1, 1, 1), proj, P, col_r, col_k,
                     col_v, col_a, zdec, PZ, w0, a0, decay_scale, cu_q, blocks, R, H, vdim, cut),
      "gdelta_chunk");
  if (rc != GB_OK) return rc;
  return delta_chunk::launch_walk<true>("gdelta_chunk", blocks, cu_q, slots, state, state_stride, R, walked, H, dim, vdim, cut, numbers, out,
                                         stream);
}

// One token per request (row t of the batch is request t). Takes vdim <= 256.
GB_EXPORT int gb_gdelta_decode(const float* proj, int P, int col_r, int col_k, int col_v, int col_a, int col_g,
                               const float* zdec, int PZ, const float* w0, const float* a0, float decay_scale,
                               const float* norm_w, float eps, const int32_t* slots, float* state, long long state_stride,
                               int R, int H, int dim, int vdim, void* out, int out_dtype, cudaStream_t stream) {
  if (R <= 0) return GB_OK;
  if (H < 1 || dim < 1 || vdim < 1) return gb::fail(GB_BAD_ARGUMENT, "gdelta_decode: sizes");
  if (vdim > 256) return gb::fail(GB_UNSUPPORTED, "gdelta_decode: %d value channels per head (at most 256)", vdim);
  const int threads = (vdim + 31) / 32 * 32;
  const size_t smem = (size_t)(5 * dim + vdim) * sizeof(float);
  return GB_DISPATCH_DTYPE(out_dtype, OT, [&]() -> int {
    return by_dim(dim, "gdelta_decode", [&](auto maxd) -> int {
      return gb::check_pdl_launch(
          gb::launch_pdl(gdelta_decode_kernel<decltype(maxd)::value, OT>, dim3(H, R), dim3(threads), smem, stream,
                         dim3(1, 1, 1), proj, P, col_r, col_k, col_v, col_a, col_g, zdec, PZ, w0, a0, decay_scale, norm_w, eps,
                         slots, state, state_stride, H, dim, vdim, (OT*)out),
          "gdelta_decode");
    });
  });
}
