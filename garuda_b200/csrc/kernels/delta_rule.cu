// The gated delta rule with a decay per key channel: a recurrent mixer whose state per request and
// head is a matrix S [dim, vdim] in 32-bit, with a short causal convolution in front of its
// query, key and value projections. Per token, in this order:
//     S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// with k and q unit vectors per head (q also times dim^-1/2), beta = sigmoid(.), and
// g = exp(-exp(A_h) softplus(a + dt_bias)) per head and key channel.
//
// Kernels, all 32-bit arithmetic:
//   delta_prepare     a block per token: convolution over the step's rows and the request's kept
//                     last inputs, SiLU, unit vectors, decays, beta
//   delta_conv_state  a request's kept last inputs after the step
//   delta_recurrence  the columns of S are independent of one another, so a request's tokens are
//                     walked in order with no exchange between columns: eight threads share a
//                     column (every eighth row each, in registers) and exchange two sums per token
//                     by shuffles; the step's q, k and g rows come through shared memory a few
//                     tokens at a time
//   delta_out         per head: o / rms(o) * weight * sigmoid(gate)
//   delta_decode      all of the above for steps of one token per request, one block per
//                     (request, head)
//   delta_chunk_factors, delta_chunk::walk
//                     the same for long stretches of tokens in a bfloat16 run, 32 tokens at a time
//                     (delta_chunk.cuh)
// In the token-by-token kernels a token's result depends on its request's earlier tokens only through the
// state, which is carried bit for bit: cutting a prompt anywhere gives the same numbers. The chunked ones add the same
// terms in another order, so there a cut moves the last bits.
#include <type_traits>

#include "common.cuh"
#include "delta_chunk.cuh"

namespace {

constexpr int MAX_TAPS = 8;

__device__ __forceinline__ float silu(float z) { return gb::divide(z, 1.0f + expf(-z)); }
__device__ __forceinline__ float sigmoid(float z) { return gb::over(1.0f + expf(-z)); }
__device__ __forceinline__ float softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// Input of channel c at `lag` tokens before token t (index j within its request's rows of this step):
// from the step's rows, or from the request's kept inputs [taps - 1, C] (oldest first).
__device__ __forceinline__ float conv_input(const float* __restrict__ proj, int P, int t, int j, int lag, int c,
                                            const float* __restrict__ kept, int C, int taps) {
  if (j - lag >= 0) return proj[(size_t)(t - lag) * P + c];
  if (kept == nullptr) return 0.f;
  return kept[(size_t)(taps - 1 + j - lag) * C + c];
}

// proj [T, P]: columns q (G dim) | k (G dim) | v (H vdim) | beta (H); the first C = 2 G dim + H vdim are
// the convolved channels. second [T, P2]: its first H dim columns are the decay's pre-activation.
// prep [T, W]: q^ (G dim) | k^ (G dim) | v (H vdim) | g (H dim) | beta (H).
template <typename WT>
__global__ void __launch_bounds__(256)
delta_prepare_kernel(const float* __restrict__ proj, int P, const float* __restrict__ second, int P2,
                     const WT* __restrict__ conv_w, int taps, const float* __restrict__ conv_state,
                     long long state_stride, const WT* __restrict__ a_log, const WT* __restrict__ dt_bias,
                     const int32_t* __restrict__ token_req, const int32_t* __restrict__ cu_q,
                     const int32_t* __restrict__ slots, float* __restrict__ prep, int W, int H, int G, int dim,
                     int vdim, int per_head, int below) {
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  extern __shared__ float act[];        // [C]
  const int t = blockIdx.x;
  const int r = token_req[t];
  if (below > 0 && cu_q[r + 1] - cu_q[r] >= below) return;      // the chunked kernels' request
  const int j = t - cu_q[r];
  const int slot = slots[r];
  const float* kept = slot >= 0 ? conv_state + (size_t)slot * state_stride : nullptr;
  const int C = 2 * G * dim + H * vdim;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float acc = 0.f;
    for (int tap = 0; tap < taps; ++tap)      // the last column weighs the current token
      acc = fmaf(gb::to_float<WT>(conv_w[(size_t)c * taps + tap]), conv_input(proj, P, t, j, taps - 1 - tap, c, kept, C, taps), acc);
    act[c] = silu(acc);
  }
  __syncthreads();
  float* out = prep + (size_t)t * W;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  // unit vectors: 2 G heads of dim channels, a warp each
  for (int hh = warp; hh < 2 * G; hh += warps) {
    const float* v = act + hh * dim;
    float ss = 0.f;
    for (int d = lane; d < dim; d += 32) ss = fmaf(v[d], v[d], ss);
    ss = gb::warp_sum(ss);
    float inv = 1.0f / sqrtf(ss + 1e-6f);
    if (hh < G) inv *= 1.0f / sqrtf((float)dim);
    for (int d = lane; d < dim; d += 32) out[hh * dim + d] = v[d] * inv;
  }
  const int off_v = 2 * G * dim, off_g = off_v + H * vdim, off_b = off_g + H * dim;
  for (int c = threadIdx.x; c < H * vdim; c += blockDim.x) out[off_v + c] = act[off_v + c];
  const float* a = second + (size_t)t * P2;
  // per_head: one decay for all key channels of a head (its pre-activation and bias are per head)
  for (int c = threadIdx.x; c < H * dim; c += blockDim.x) {
    const float rate = expf(gb::to_float<WT>(a_log[c / dim]));
    const int j = per_head ? c / dim : c;
    out[off_g + c] = expf(-rate * softplus(a[j] + gb::to_float<WT>(dt_bias[j])));
  }
  for (int h = threadIdx.x; h < H; h += blockDim.x) out[off_b + h] = sigmoid(proj[(size_t)t * P + C + h]);
}

// grid (R, ceil(C / 256)): the request's last taps - 1 inputs after this step, oldest first. A
// thread owns a channel and walks its entries in ascending order, reading only entries above
// the one it writes.
__global__ void __launch_bounds__(256)
delta_conv_state_kernel(const float* __restrict__ proj, int P, float* __restrict__ conv_state, long long state_stride,
                        const int32_t* __restrict__ cu_q, const int32_t* __restrict__ slots, int C, int taps) {
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  const int r = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const int slot = slots[r];
  if (c >= C || slot < 0) return;
  const int t0 = cu_q[r], n = cu_q[r + 1] - t0;
  float* kept = conv_state + (size_t)slot * state_stride;
  const int keep = taps - 1;
  for (int i = 0; i < keep; ++i) {
    const int src = i + n;                  // index in (kept inputs, then the step's rows)
    kept[(size_t)i * C + c] = src < keep ? kept[(size_t)src * C + c] : proj[(size_t)(t0 + src - keep) * P + c];
  }
}

constexpr int CHUNK = 8;
constexpr int SPLIT = 8;        // threads that share a column of S: thread `sub` holds the rows d with d % 8 == sub
constexpr int REC_THREADS = 128, REC_COLS = REC_THREADS / SPLIT;

// grid (H, R, ceil(vdim / 16)), 128 threads: 16 columns of S, eight threads a column. Each of the
// eight sums its rows in ascending order and the eight are added as a tree, ((0 + 1) + (2 + 3)) +
// ((4 + 5) + (6 + 7)): the same sums, in the same order, as the eight interleaved partial sums of
// the one-token kernel below. Everything a token needs (q^, k^, g, the block's values, beta)
// comes through shared memory, eight tokens at a time in two buffers: the next eight are on their
// way while these are walked. EXACT: dim == MAXD, no row of a thread is beyond the head's.
template <int MAXD, bool EXACT>
__global__ void __launch_bounds__(REC_THREADS)
delta_recurrence_kernel(const float* __restrict__ prep, int W, const int32_t* __restrict__ cu_q,
                        const int32_t* __restrict__ slots, float* __restrict__ state, long long state_stride, int H,
                        int G, int dim, int vdim, int below, float* __restrict__ out) {
  gb::pdl_wait();
  if (below > 0 && cu_q[blockIdx.y + 1] - cu_q[blockIdx.y] >= below) return;      // the chunked kernels' request
  constexpr int MINE = MAXD / SPLIT;
  extern __shared__ __align__(16) float stage[];      // 2 x [CHUNK][3 SPLIT per + 32 + 4]
  // a thread's rows, rounded up to whole 16-byte pieces, and one piece more: the four slices start
  // in different banks and are read four values at a time
  const int per = ((dim + SPLIT - 1) / SPLIT + 3) / 4 * 4 + 4;
  const int tok_floats = 3 * SPLIT * per + REC_COLS + 4;      // a multiple of four: every slice starts on 16 bytes
  const int h = blockIdx.x, r = blockIdx.y;
  const int sub = threadIdx.x % SPLIT;
  const int col0 = blockIdx.z * REC_COLS, mycol = threadIdx.x / SPLIT, col = col0 + mycol;
  const bool active = col < vdim;
  const int slot = slots[r];
  const int t0 = cu_q[r], t1 = cu_q[r + 1];
  const int kvh = h / (H / G);
  const int off_q = kvh * dim, off_k = G * dim + kvh * dim, off_v = 2 * G * dim + h * vdim + col0;
  const int off_g = 2 * G * dim + H * vdim + h * dim, off_b = off_g - h * dim + H * dim + h;
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
      const float* row = prep + (size_t)(c0 + tt) * W;
      float* to = dst + tt * tok_floats + (d % SPLIT) * per + d / SPLIT;
      delta_chunk::copy_4(to, row + off_q + d);
      delta_chunk::copy_4(to + SPLIT * per, row + off_k + d);
      delta_chunk::copy_4(to + 2 * SPLIT * per, row + off_g + d);
    }
    for (int i = threadIdx.x; i < n * (ncols + 1); i += REC_THREADS) {
      const int tt = i / (ncols + 1), c = i % (ncols + 1);
      const float* row = prep + (size_t)(c0 + tt) * W;
      float* to = dst + tt * tok_floats + 3 * SPLIT * per;
      if (c < ncols) delta_chunk::copy_4(to + c, row + off_v + c);
      else delta_chunk::copy_4(to + REC_COLS, row + off_b);
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
      const float* sq = tok + sub * per;
      const float* sk = sq + SPLIT * per;
      const float* sg = sk + SPLIT * per;
      const float v = active ? tok[3 * SPLIT * per + mycol] : 0.f;
      const float beta = tok[3 * SPLIT * per + REC_COLS];
      float acc = 0.f;
      float kk[MINE];
#pragma unroll
      for (int i4 = 0; i4 < MINE; i4 += 4) {
        if (!EXACT && i4 * SPLIT >= dim) break;         // pieces beyond the head's rows are not in shared memory
        const float4 g4 = *reinterpret_cast<const float4*>(sg + i4);
        const float4 k4 = *reinterpret_cast<const float4*>(sk + i4);
        const float gg[4] = {g4.x, g4.y, g4.z, g4.w};
        kk[i4] = k4.x, kk[i4 + 1] = k4.y, kk[i4 + 2] = k4.z, kk[i4 + 3] = k4.w;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (EXACT || (i4 + j) * SPLIT + sub < dim) {
            S[i4 + j] *= gg[j];
            acc = fmaf(S[i4 + j], kk[i4 + j], acc);
          }
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      acc += __shfl_xor_sync(0xffffffffu, acc, 4);
      const float u = beta * (v - acc);
      float o = 0.f;
#pragma unroll
      for (int i4 = 0; i4 < MINE; i4 += 4) {
        if (!EXACT && i4 * SPLIT >= dim) break;
        const float4 q4 = *reinterpret_cast<const float4*>(sq + i4);
        const float qq[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (EXACT || (i4 + j) * SPLIT + sub < dim) {
            S[i4 + j] = fmaf(kk[i4 + j], u, S[i4 + j]);
            o = fmaf(S[i4 + j], qq[j], o);
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

// What the walk of delta_chunk.cuh needs of a chunk and a head: convolution, SiLU, unit vectors, decays and beta as in
// delta_prepare, then, with D_i the product of the decays up to token i,
//     L_ij = beta_i sum_d k_i k_j D_i / D_j (j < i),   B_ij = sum_d q_i k_j D_i / D_j (j <= i)
//     W = (I + L)^-1 beta (D k),   VP = (I + L)^-1 beta v,   Q = D q - B W,   OP = B VP,   K1_j = k_j D_last / D_j
// The quotients D_i / D_j are products of decays between j and i, and the triangular system is solved by substitution: both in blocks
// of 8 tokens (delta_chunk.cuh), on the tensor cores off the diagonal and in 32-bit multiply-adds on it.
// What bounds it: the chunk's rows and results (2,048 tokens of 16 heads of 128 x 128 read 68 MB and write 84, 23 us), and the latency of
// its six phases, three blocks an SM. With dots of all pairs by running products and a thread per column in the substitution
// (33,000 of a block's 84,000 cycles, for the rows of L and B, which every warp read from shared memory for itself) 124 us, now 118.
// grid (numbers, H), 256 threads; at most four taps.
template <int DIM>
struct FactorsSmem {
  delta_chunk::Lower L, B;
  // [tokens][DIM + 8] each. k and q: then decayed on from their block's start; g: decays (kept_decay), keys decayed on to their block's end,
  // values
  float k[delta_chunk::C * (DIM + 8)], q[delta_chunk::C * (DIM + 8)], g[delta_chunk::C * (DIM + 8)];
  float2 through[delta_chunk::NB * DIM];         // whole blocks' decays (delta_chunk::Product)
  float beta[delta_chunk::C];
};
template <int DIM, typename WT>
__global__ void __launch_bounds__(256, 3)
delta_chunk_factors_kernel(const float* __restrict__ proj, int P, const float* __restrict__ second, int P2,
                           const WT* __restrict__ conv_w, int taps, const float* __restrict__ conv_state, long long conv_stride,
                           const WT* __restrict__ a_log, const WT* __restrict__ dt_bias, const int32_t* __restrict__ cu_q,
                           const int32_t* __restrict__ slots, float* __restrict__ blocks, int R, int H, int G, int vdim, int per_head,
                           int cut) {
  using namespace delta_chunk;
  using delta_chunk::C;
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  constexpr int LD = DIM + 8, VEC = DIM / 32;
  extern __shared__ __align__(16) unsigned char raw[];
  FactorsSmem<DIM>& sm = *reinterpret_cast<FactorsSmem<DIM>*>(raw);
  float *sk = sm.k, *sq = sm.q, *sg = sm.g, *beta = sm.beta;
  Lower &L = sm.L, &B = sm.B;
  const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int r, first, n, at;
  if (!find_chunk(blockIdx.x, cu_q, R, cut, r, first, n, at)) return;
  const Layout lay{DIM, vdim, 0};
  float* block = blocks + ((size_t)blockIdx.x * H + h) * lay.floats();
  const int slot = slots[r], kvh = h / (H / G), CH = 2 * G * DIM + H * vdim;
  const float* kept = slot >= 0 ? conv_state + (size_t)slot * conv_stride : nullptr;
  // The chunk's rows of q, k and the decays' pre-activations come into their places in shared memory all at once, 16 bytes a copy where
  // rows start on 16 bytes (fetched by the threads that use them, eight numbers ahead, they were a third of this kernel's time).
  {
    auto rows = [&](float* to, const float* from, int pitch) {
      if (pitch % 4 == 0 && ((uintptr_t)from & 15) == 0) {
        for (int i = tid; i < n * (DIM / 4); i += 256)
          copy_16(to + i / (DIM / 4) * LD + i % (DIM / 4) * 4, from + (size_t)(i / (DIM / 4)) * pitch + i % (DIM / 4) * 4);
      } else {
        for (int i = tid; i < n * DIM; i += 256) delta_chunk::copy_4(to + i / DIM * LD + i % DIM, from + (size_t)(i / DIM) * pitch + i % DIM);
      }
    };
    const float* q0 = proj + (size_t)first * P + kvh * DIM;
    rows(sq, q0, P);
    rows(sk, q0 + G * DIM, P);
    if (!per_head) rows(sg, second + (size_t)first * P2 + h * DIM, P2);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // Convolution and SiLU of a channel's tokens from i1 on, TURN of them: `in` their inputs, x those in front, the last first
  auto weights = [&](int ch, float (&w)[4]) {              // by lag
#pragma unroll
    for (int lag = 0; lag < 4; ++lag) w[lag] = lag < taps ? gb::to_float<WT>(conv_w[(size_t)ch * taps + taps - 1 - lag]) : 0.f;
  };
  auto in_front = [&](int ch, int i1, float (&x)[3]) {
#pragma unroll
    for (int lag = 1; lag < 4; ++lag) x[lag - 1] = lag < taps && i1 < n ? conv_input(proj, P, first + i1, at + i1, lag, ch, kept, CH, taps) : 0.f;
  };
  auto convolve = [&](const float (&w)[4], float (&x)[3], int i1, const auto& in, auto&& take) {
    constexpr int TURN = sizeof(in) / sizeof(float);
#pragma unroll
    for (int e = 0; e < TURN; ++e) {
      // (an input further back than the taps reach must not count: with a weight of zero an infinity would)
      float acc = taps > 3 ? fmaf(w[3], x[2], 0.f) : 0.f;
      if (taps > 2) acc = fmaf(w[2], x[1], acc);
      if (taps > 1) acc = fmaf(w[1], x[0], acc);
      acc = fmaf(w[0], in[e], acc);
      x[2] = x[1], x[1] = x[0], x[0] = in[e];
      take(i1 + e, i1 + e < n ? silu(acc) : 0.f);
    }
  };
  const float rate = expf(gb::to_float<WT>(a_log[h]));
  if (tid < C) beta[tid] = tid < n ? sigmoid(proj[(size_t)(first + tid) * P + CH + h]) : 0.f;
  if (per_head) {
    // one decay for all key channels: every thread's warp makes one token's at a time
    for (int t = warp; t < C; t += 8) {
      const float g = t < n ? kept_decay(-rate * softplus(second[(size_t)(first + t) * P2 + h] + gb::to_float<WT>(dt_bias[h]))) : 0.f;
      for (int d = lane; d < DIM; d += 32) sg[t * LD + d] = g;
    }
  } else {
    const float bias = gb::to_float<WT>(dt_bias[h * DIM + tid % DIM]);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll 4
    for (int t = tid / DIM; t < C; t += 256 / DIM) {
      float* a = sg + t * LD + tid % DIM;
      *a = t < n ? kept_decay(-rate * softplus(*a + bias)) : 0.f;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int c = tid; c < 2 * DIM; c += 256) {               // in place: a thread owns its channels' columns
    const bool query = c < DIM;
    float* col = query ? sq + c : sk + c - DIM;
    const int ch = query ? kvh * DIM + c : (G + kvh) * DIM + c - DIM;
    float w[4], x[3], in[16];
    weights(ch, w), in_front(ch, 0, x);
#pragma unroll
    for (int i0 = 0; i0 < C; i0 += 16) {
#pragma unroll
      for (int e = 0; e < 16; ++e) in[e] = i0 + e < n ? col[(i0 + e) * LD] : 0.f;
      convolve(w, x, i0, in, [&](int i, float v) { col[i * LD] = v; });
    }
  }
  __syncthreads();
#pragma unroll
  for (int row = warp; row < 2 * C; row += 8) {
    float* v = row < C ? sq + row * LD : sk + (row - C) * LD;
    float x[VEC], ss = 0.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e) x[e] = v[lane + 32 * e], ss = fmaf(x[e], x[e], ss);
    ss = gb::warp_sum(ss);
    // queries over the root of DIM as well: of 64 an eighth, of 128 a sixteenth times the root of two
    const bool query = row < C;
    const float2 inv = one_over_root((ss + 1e-6f) * (query && DIM == 128 ? 0.5f : 1.f));
    const float by = query ? (DIM == 128 ? 0.0625f : 0.125f) : 1.f;
#pragma unroll
    for (int e = 0; e < VEC; ++e) v[lane + 32 * e] = by * fmaf(x[e], inv.x, x[e] * inv.y);
  }
  __syncthreads();
  {
    // L and B on the diagonal: a warp has four keys j, each decayed on from token to token up to its block's end
    const int j0 = warp * 4, j1 = (warp | 1) * 4 + 4, d0 = lane * VEC;
    pair_t p[4][VEC / 2];
    auto row = [&](const float* m, int i, pair_t (&x)[VEC / 2]) {
      if (VEC == 4) {
        const pair2_t f = *reinterpret_cast<const pair2_t*>(m + i * LD + d0);
        x[0] = f.a, x[VEC / 2 - 1] = f.b;
      } else {
        x[0] = *reinterpret_cast<const pair_t*>(m + i * LD + d0);
      }
    };
    auto decays = [&](int i, pair_t (&x)[VEC / 2]) {
      row(sg, i, x);
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
    auto keep = [&](int i, float (&v)[8]) {
      const float sum = sum_of_eight(v, lane);
      const int which = lane >> 2, j = j0 + (which & 3);
      if ((lane & 3) == 0) {
        if (which < 4) {
          if (j < i) L.on[j >> 3][(j & 7) * 8 + (i & 7)] = beta[i] * sum;
        } else if (j <= i) {
          B.on[j >> 3][(j & 7) * 8 + (i & 7)] = sum;
        }
      }
    };
#pragma unroll
    for (int ii = 0; ii < 4; ++ii) {       // the tokens of the four keys themselves
      const int i = j0 + ii;
      pair_t g[VEC / 2], k[VEC / 2], q[VEC / 2];
      decays(i, g), row(sk, i, k), row(sq, i, q);
      float v[8];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
        for (int e = 0; e < VEC / 2; ++e) p[jj][e] = jj < ii ? mul2(p[jj][e], g[e]) : k[e];
        v[jj] = jj < ii ? dot(p[jj], k) : 0.f;
        v[4 + jj] = jj <= ii ? dot(p[jj], q) : 0.f;
      }
      keep(i, v);
    }
#pragma unroll 2
    for (int i = j0 + 4; i < j1; ++i) {
      pair_t g[VEC / 2], k[VEC / 2], q[VEC / 2];
      decays(i, g), row(sk, i, k), row(sq, i, q);
      float v[8];
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
        for (int e = 0; e < VEC / 2; ++e) p[jj][e] = mul2(p[jj][e], g[e]);
        v[jj] = dot(p[jj], k);
        v[4 + jj] = dot(p[jj], q);
      }
      keep(i, v);
    }
  }
  __syncthreads();
  // decayed on within a block of tokens: queries and keys from its start, and keys, in the decays' place, to its end
  for (int i = tid; i < NB * DIM; i += 256) {
    const int c = i % DIM, at0 = i / DIM * 8 * LD + c;
    float g[8], k[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) g[t] = sg[at0 + t * LD], k[t] = sk[at0 + t * LD];
    Product on, behind;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      on.by(whole_decay(g[t]));
      sq[at0 + t * LD] = on.of(sq[at0 + t * LD]);
      sk[at0 + t * LD] = on.of(k[t]);
    }
    sm.through[i] = on.both();
#pragma unroll
    for (int t = 7; t >= 0; --t) {
      sg[at0 + t * LD] = behind.of(k[t]);
      behind.by(whole_decay(g[t]));
    }
  }
  __syncthreads();
  for (int task = warp; task < BELOW; task += 8) {
    const int bi = task < 1 ? 1 : task < 3 ? 2 : 3, bj = task - below(bi, 0);
    float acc[4];
    block_below<DIM, LD>(acc, sq, sk, sg, sm.through, bi, bj, lane);
    const float b = beta[bi * 8 + (lane >> 2)];
    B.off[task][lane] = split_pair(acc[0], acc[1]);
    L.off[task][lane] = split_pair(b * acc[2], b * acc[3]);
  }
  for (int i = tid; i < NB * DIM; i += 256) {              // K1, and the chunk's whole decay
    const int c = i % DIM, bj = i / DIM;
    Product behind;
    float x[8];
#pragma unroll
    for (int b = NB - 1; b > 0; --b)
      if (b > bj) behind.by(sm.through[b * DIM + c]);
#pragma unroll
    for (int t = 0; t < 8; ++t) x[t] = behind.of(sg[(bj * 8 + t) * LD + c]);
    float4* to = reinterpret_cast<float4*>(block + lay.k1(bj * 8, c));
    to[0] = make_float4(x[0], x[1], x[2], x[3]), to[1] = make_float4(x[4], x[5], x[6], x[7]);
    if (bj == 0) {
      behind.by(sm.through[c]);
      block[lay.last() + c] = behind.value();
    }
  }
  __syncthreads();
  // The substitution: the keys' columns, and the values' up to DIM at a time, which are convolved into the decays' place
  const int g = lane >> 2, tig = lane & 3;
  auto columns = [&](auto keys, int col0, const float* from, float* vp, float* op) {
    float take[NB][4], more[NB][4];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int e = 0; e < 4; ++e) take[b][e] = more[b][e] = 0.f;
    Product front[2];         // keys: D, as the blocks in front make it
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const float beta2[2] = {beta[b * 8 + 2 * tig], beta[b * 8 + 2 * tig + 1]};
      float x[4], y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[e] = from[(b * 8 + 2 * tig + (e & 1)) * LD + g + 8 * (e >> 1)];
        if (keys) x[e] = front[e >> 1].of(x[e]);
      }
      on_diagonal(L.on[b], B.on[b], lane, take[b], more[b], [&](int e) { return fmaf(beta2[e & 1], x[e], take[b][e]); });
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = fmaf(beta2[e & 1], x[e], take[b][e]);
      if (b + 1 < NB) below_diagonal(L, B, b, lane, y, take, more);
      if (keys) {
        store_tile_rows(block, lay, b * 8, col0, lane, y);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = front[e >> 1].of(sq[(b * 8 + 2 * tig + (e & 1)) * LD + col0 + g + 8 * (e >> 1)]) - more[b][e];
        store_tile_rows(block, lay, C + b * 8, col0, lane, x);
        front[0].by(sm.through[b * DIM + col0 + g]), front[1].by(sm.through[b * DIM + col0 + g + 8]);
      } else {
        store_tile_columns(vp, col0, b, lane, y);
        store_tile_columns(op, col0, b, lane, more[b]);
      }
    }
  };
  for (int v0 = 0; v0 < vdim; v0 += DIM) {
    constexpr int EACH = C * DIM / 256;            // a thread's tokens of a channel
    const int vc = tid % DIM, v1 = tid / DIM * EACH, ch = 2 * G * DIM + h * vdim + v0 + vc;
    if (v0 > 0) __syncthreads();
    if (v0 + vc < vdim) {
      float w[4], x[3], in[EACH];
      weights(ch, w), in_front(ch, v1, x);
#pragma unroll
      for (int e = 0; e < EACH; ++e) in[e] = v1 + e < n ? proj[(size_t)(first + v1 + e) * P + ch] : 0.f;
      convolve(w, x, v1, in, [&](int i, float v) { sg[i * LD + vc] = v; });
    }
    if (v0 == 0 && warp * 16 < DIM) columns(std::true_type{}, warp * 16, sk + warp * 16, nullptr, nullptr);
    __syncthreads();
    if (v0 + warp * 16 < vdim && warp * 16 < DIM)
      columns(std::false_type{}, v0 + warp * 16, sg + warp * 16, block + lay.vp(), block + lay.op());
  }
}

// out[t][h] = o / sqrt(mean(o^2) + eps) * w * act(gate), act = sigmoid or SiLU; w [vdim] shared by the heads or [H vdim]. gate:
// columns gate_off .. of `second`. A warp per (token, head), four a block; everything a lane needs (every 32nd channel, N of them) is asked
// for before anything is used. Bound by memory: 2,048 tokens of 16 heads of 128 read 33 MB and write 8 (a block per token whose warps
// took the heads in turn, gates asked for after the sum: 27 us; now 12.7).
template <int N, typename WT, typename OT>
__global__ void __launch_bounds__(128)
delta_out_kernel(const float* __restrict__ o, const float* __restrict__ second, int P2, int gate_off,
                 const WT* __restrict__ w, float eps, OT* __restrict__ out, int H, int vdim, int silu_gate,
                 int w_per_head, long long rows) {
  gb::pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const long long at = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (at >= rows) return;
  const int h = (int)(at % H);
  const size_t t = (size_t)(at / H);
  const WT* wh = w_per_head ? w + (size_t)h * vdim : w;
  float weight[N];
#pragma unroll
  for (int i = 0; i < N; ++i) weight[i] = lane + 32 * i < vdim ? gb::to_float<WT>(wh[lane + 32 * i]) : 0.f;
  gb::pdl_wait();
  const float* row = o + (size_t)at * vdim + lane;
  const float* gate = second + t * P2 + gate_off + h * vdim + lane;
  float x[N], g[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    x[i] = lane + 32 * i < vdim ? row[32 * i] : 0.f;
    g[i] = lane + 32 * i < vdim ? gate[32 * i] : 0.f;
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) ss = fmaf(x[i], x[i], ss);
  const float scale = 1.0f / sqrtf(gb::warp_sum(ss) / (float)vdim + eps);
  OT* to = out + (size_t)at * vdim + lane;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (lane + 32 * i < vdim) to[32 * i] = gb::from_float<OT>((x[i] * scale) * weight[i] * (silu_gate ? silu(g[i]) : sigmoid(g[i])));
}

// the same for any vdim: a lane's channels one after another
template <typename WT, typename OT>
__global__ void __launch_bounds__(128)
delta_out_any_kernel(const float* __restrict__ o, const float* __restrict__ second, int P2, int gate_off,
                     const WT* __restrict__ w, float eps, OT* __restrict__ out, int H, int vdim, int silu_gate,
                     int w_per_head, long long rows) {
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long at = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (at >= rows) return;
  const int h = (int)(at % H);
  const size_t t = (size_t)(at / H);
  const float* row = o + (size_t)at * vdim;
  const float* gate = second + t * P2 + gate_off + h * vdim;
  float ss = 0.f;
  for (int c = lane; c < vdim; c += 32) ss = fmaf(row[c], row[c], ss);
  const float scale = 1.0f / sqrtf(gb::warp_sum(ss) / (float)vdim + eps);
  const WT* wh = w_per_head ? w + (size_t)h * vdim : w;
  for (int c = lane; c < vdim; c += 32)
    out[(size_t)at * vdim + c] = gb::from_float<OT>((row[c] * scale) * gb::to_float<WT>(wh[c]) * (silu_gate ? silu(gate[c]) : sigmoid(gate[c])));
}

// A step of one token per request: grid (H, R), vdim threads (a column of S each, rounded up to a
// warp). Every block convolves the channels of its own head (its key/value head's q and k, its v),
// so nothing is exchanged between blocks; block h == 0 .. G - 1 also writes nothing extra: the kept
// inputs are shifted by a kernel behind this one. The state column lives in registers for the one
// token: read, decayed, updated, written.
template <int MAXD, typename WT, typename OT>
__global__ void __launch_bounds__(256)
delta_decode_kernel(const float* __restrict__ proj, int P, const float* __restrict__ second, int P2,
                    const WT* __restrict__ conv_w, int taps, const float* __restrict__ conv_state, long long conv_stride,
                    const WT* __restrict__ a_log, const WT* __restrict__ dt_bias, const WT* __restrict__ norm_w, float eps,
                    const int32_t* __restrict__ slots, float* __restrict__ state, long long state_stride, int H, int G,
                    int dim, int vdim, OT* __restrict__ out, int per_head, int gate_off, int silu_gate) {
  gb::pdl_launch_dependents();
  gb::pdl_wait();
  extern __shared__ float sm[];          // q^[dim], k^[dim], g[dim], scratch[32], o[vdim]
  float* sq = sm;
  float* sk = sm + dim;
  float* sg = sm + 2 * dim;
  float* scratch = sm + 3 * dim;
  const int h = blockIdx.x, t = blockIdx.y;         // one token per request: row t is request t
  const int slot = slots[t];
  const int kvh = h / (H / G);
  const int C = 2 * G * dim + H * vdim;
  const float* kept = slot >= 0 ? conv_state + (size_t)slot * conv_stride : nullptr;
  auto conv = [&](int c) {
    float acc = 0.f;
    for (int tap = 0; tap < taps; ++tap)
      acc = fmaf(gb::to_float<WT>(conv_w[(size_t)c * taps + tap]), conv_input(proj, P, t, 0, taps - 1 - tap, c, kept, C, taps), acc);
    return silu(acc);
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int d = threadIdx.x; d < dim; d += blockDim.x) {
    sq[d] = conv(kvh * dim + d);
    sk[d] = conv(G * dim + kvh * dim + d);
    const int c = per_head ? h : h * dim + d;
    sg[d] = expf(-expf(gb::to_float<WT>(a_log[h])) * softplus(second[(size_t)t * P2 + c] + gb::to_float<WT>(dt_bias[c])));
  }
  __syncthreads();
  // unit vectors: warp 0 the query, warp 1 (or 0 again) the key
  for (int which = warp; which < 2; which += warps) {
    float* v = which == 0 ? sq : sk;
    float ss = 0.f;
    for (int d = lane; d < dim; d += 32) ss = fmaf(v[d], v[d], ss);
    ss = gb::warp_sum(ss);
    float inv = 1.0f / sqrtf(ss + 1e-6f);
    if (which == 0) inv *= 1.0f / sqrtf((float)dim);
    __syncwarp();
    for (int d = lane; d < dim; d += 32) v[d] *= inv;
  }
  __syncthreads();
  const int col = threadIdx.x;
  const bool active = col < vdim;
  float o_val = 0.f;
  if (active) {
    const float v = conv(2 * G * dim + h * vdim + col);
    const float beta = sigmoid(proj[(size_t)t * P + C + h]);
    float* S_g = slot >= 0 ? state + (size_t)slot * state_stride + (size_t)h * dim * vdim + col : nullptr;
    float S[MAXD];
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
      if (d < dim) {
        S[d] = (S_g != nullptr ? S_g[(size_t)d * vdim] : 0.f) * sg[d];
        acc[d & 7] = fmaf(S[d], sk[d], acc[d & 7]);
      }
    // the tree the kernel for longer steps adds its eight threads' sums by
    const float u = beta * (v - (((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]))));
    float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < MAXD; ++d)
      if (d < dim) {
        S[d] = fmaf(sk[d], u, S[d]);
        o[d & 7] = fmaf(S[d], sq[d], o[d & 7]);
        if (S_g != nullptr) S_g[(size_t)d * vdim] = S[d];
      }
    o_val = ((o[0] + o[1]) + (o[2] + o[3])) + ((o[4] + o[5]) + (o[6] + o[7]));
  }
  // the head's RMS over vdim, the weight and the output gate; the sum of squares in the order the
  // kernel for longer steps takes it (a lane's channels in ascending order, then the warp's tree),
  // so that a token's result is the same bits whichever kernel ran it
  float* so = scratch + 32;            // [vdim]
  if (active) so[col] = o_val;
  __syncthreads();
  float ss = 0.f;
  for (int c = lane; c < vdim; c += 32) ss = fmaf(so[c], so[c], ss);
  const float scale = 1.0f / sqrtf(gb::warp_sum(ss) / (float)vdim + eps);
  if (active) {
    const float gate = second[(size_t)t * P2 + gate_off + h * vdim + col];
    out[((size_t)t * H + h) * vdim + col] =
        gb::from_float<OT>((o_val * scale) * gb::to_float<WT>(norm_w[col]) * (silu_gate ? silu(gate) : sigmoid(gate)));
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

int check_sizes(const char* what, int H, int G, int dim, int vdim, int taps) {
  if (H < 1 || G < 1 || H % G) return gb::fail(GB_BAD_ARGUMENT, "%s: %d heads for %d key heads", what, H, G);
  if (dim < 1 || vdim < 1) return gb::fail(GB_BAD_ARGUMENT, "%s: head sizes %d and %d", what, dim, vdim);
  if (taps < 1 || taps > MAX_TAPS) return gb::fail(GB_UNSUPPORTED, "%s: %d taps (1 to %d)", what, taps, MAX_TAPS);
  return GB_OK;
}

}  // namespace

// state_stride, conv_stride: floats between two slots' states. below (of delta_prepare and delta_recurrence): only requests
// with fewer tokens in the step than this (0: all).
GB_EXPORT int gb_delta_prepare(const float* proj, int P, const float* second, int P2, const void* conv_w, int w_dtype,
                               int taps, const float* conv_state, long long conv_stride, const void* a_log,
                               const void* dt_bias, const int32_t* token_req, const int32_t* cu_q, const int32_t* slots,
                               float* prep, int W, int T, int H, int G, int dim, int vdim, int per_head,
                               int below, cudaStream_t stream) {
  if (T <= 0) return GB_OK;
  int rc = check_sizes("delta_prepare", H, G, dim, vdim, taps);
  if (rc != GB_OK) return rc;
  const int C = 2 * G * dim + H * vdim;
  if (P < C + H || P2 < (per_head ? H : H * dim) || W != C + H * dim + H)
    return gb::fail(GB_BAD_ARGUMENT, "delta_prepare: row widths");
  const size_t smem = (size_t)C * sizeof(float);
  constexpr size_t kMostSmem = 224 * 1024;      // what a block may ask for on this GPU, less some for the driver
  if (smem > kMostSmem) return gb::fail(GB_UNSUPPORTED, "delta_prepare: %d convolved channels (at most %d)", C, (int)(kMostSmem / 4));
  return GB_DISPATCH_DTYPE(w_dtype, WT, [&]() -> int {
    if (smem > 48 * 1024) {                      // beyond the default limit a kernel has to ask once
      static size_t granted = 0;                 // per weight type: this lambda is instantiated for each
      if (smem > granted) {
        const cudaError_t e = cudaFuncSetAttribute(delta_prepare_kernel<WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem);
        if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "delta_prepare: %s", cudaGetErrorString(e));
        granted = kMostSmem;
      }
    }
    return gb::check_pdl_launch(
        gb::launch_pdl(delta_prepare_kernel<WT>, dim3(T), dim3(256), smem, stream, dim3(1, 1, 1), proj, P, second, P2,
                       (const WT*)conv_w, taps, conv_state, conv_stride, (const WT*)a_log, (const WT*)dt_bias, token_req,
                       cu_q, slots, prep, W, H, G, dim, vdim, per_head, below),
        "delta_prepare");
  });
}

GB_EXPORT int gb_delta_conv_state(const float* proj, int P, float* conv_state, long long conv_stride, const int32_t* cu_q,
                                  const int32_t* slots, int R, int C, int taps, cudaStream_t stream) {
  if (R <= 0 || taps <= 1) return GB_OK;
  return gb::check_pdl_launch(gb::launch_pdl(delta_conv_state_kernel, dim3(R, (C + 255) / 256), dim3(256), 0, stream,
                                             dim3(1, 1, 1), proj, P, conv_state, conv_stride, cu_q, slots, C, taps),
                              "delta_conv_state");
}

GB_EXPORT int gb_delta_recurrence(const float* prep, int W, const int32_t* cu_q, const int32_t* slots, float* state,
                                  long long state_stride, int R, int H, int G, int dim, int vdim, int below, float* out,
                                  cudaStream_t stream) {
  if (R <= 0) return GB_OK;
  int rc = check_sizes("delta_recurrence", H, G, dim, vdim, 1);
  if (rc != GB_OK) return rc;
  const int threads = REC_THREADS, cols = REC_COLS;
  const dim3 grid(H, R, (vdim + cols - 1) / cols);
  const int per = ((dim + SPLIT - 1) / SPLIT + 3) / 4 * 4 + 4;
  const size_t smem = (size_t)2 * CHUNK * (3 * SPLIT * per + REC_COLS + 4) * sizeof(float);
  return by_dim(dim, "delta_recurrence", [&](auto maxd) -> int {
    if (smem > 48 * 1024) {     // never with these tile sizes (key widths up to 256 need 34 KB); kept for larger ones
      cudaError_t e1 = cudaFuncSetAttribute(delta_recurrence_kernel<decltype(maxd)::value, true>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      cudaError_t e2 = cudaFuncSetAttribute(delta_recurrence_kernel<decltype(maxd)::value, false>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e1 != cudaSuccess || e2 != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "delta_recurrence: shared memory");
    }
    constexpr int MAXD = decltype(maxd)::value;
    auto kernel = dim == MAXD ? delta_recurrence_kernel<MAXD, true> : delta_recurrence_kernel<MAXD, false>;
    return gb::check_pdl_launch(gb::launch_after(kernel, grid, dim3(threads), smem, stream, dim3(1, 1, 1), prep, W, cu_q,
                                               slots, state, state_stride, H, G, dim, vdim, below, out),
                                "delta_recurrence");
  });
}

// Whether the chunked kernels take these sizes, and the floats of `blocks` for a step of T tokens, `walked` requests of which have at
// least `cut` (0: they do not).
GB_EXPORT long long gb_delta_chunk_floats(int T, int walked, int H, int G, int dim, int vdim, int taps) {
  if (T <= 0 || walked <= 0 || H < 1 || H > 65535 || walked > 65535 || G < 1 || H % G || taps < 1 || taps > 4 || !delta_chunk::takes(dim, vdim)) return 0;
  return (long long)delta_chunk::chunk_numbers(T, walked) * H * delta_chunk::Layout{dim, vdim, 0}.floats();
}

// Requests of at least `cut` tokens: everything from the projected rows to the read-out o [T, H vdim] and the state. The rows
// are those of delta_prepare; walked: how many such requests the step has; blocks starts on 16 bytes.
GB_EXPORT int gb_delta_chunk(const float* proj, int P, const float* second, int P2, const void* conv_w, int w_dtype, int taps,
                             const float* conv_state, long long conv_stride, const void* a_log, const void* dt_bias,
                             const int32_t* cu_q, const int32_t* slots, float* state, long long state_stride, float* blocks, int T,
                             int R, int walked, int H, int G, int dim, int vdim, int per_head, int cut, float* out, cudaStream_t stream) {
  if (T <= 0 || R <= 0 || walked <= 0) return GB_OK;
  if (R > 65535 || gb_delta_chunk_floats(T, walked, H, G, dim, vdim, taps) == 0)
    return gb::fail(GB_UNSUPPORTED, "delta_chunk: %d heads of %d x %d, %d key heads, %d taps", H, dim, vdim, G, taps);
  const int CH = 2 * G * dim + H * vdim, numbers = delta_chunk::chunk_numbers(T, walked);
  if (P < CH + H || P2 < (per_head ? H : H * dim)) return gb::fail(GB_BAD_ARGUMENT, "delta_chunk: row widths");
  if ((uintptr_t)blocks & 15) return gb::fail(GB_BAD_ARGUMENT, "delta_chunk: blocks start on 16 bytes");
  const size_t smem = dim == 128 ? sizeof(FactorsSmem<128>) : sizeof(FactorsSmem<64>);
  const int rc = GB_DISPATCH_DTYPE(w_dtype, WT, [&]() -> int {
    auto kernel = dim == 128 ? delta_chunk_factors_kernel<128, WT> : delta_chunk_factors_kernel<64, WT>;
    static gb::OncePerDevice configured[2];      // per weight type: this lambda is instantiated for each
    if (configured[dim == 128].needed()) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "delta_chunk: %s", cudaGetErrorString(e));
      configured[dim == 128].done();
    }
    return gb::check_pdl_launch(
        gb::launch_pdl(kernel, dim3(numbers, H), dim3(256), smem, stream, dim3(1, 1, 1), proj, P, second, P2,
                       (const WT*)conv_w, taps, conv_state, conv_stride, (const WT*)a_log, (const WT*)dt_bias, cu_q, slots, blocks, R, H,
                       G, vdim, per_head, cut),
        "delta_chunk");
  });
  if (rc != GB_OK) return rc;
  return delta_chunk::launch_walk<false>("delta_chunk", blocks, cu_q, slots, state, state_stride, R, walked, H, dim, vdim, cut, numbers, out,
                                         stream);
}

GB_EXPORT int gb_delta_out(const float* o, const float* second, int P2, int gate_off, const void* w, int w_dtype,
                           float eps, void* out, int out_dtype, int T, int H, int vdim, int silu_gate, int w_per_head,
                           cudaStream_t stream) {
  if (T <= 0) return GB_OK;
  return GB_DISPATCH_DTYPE(w_dtype, WT, [&]() -> int {
    return GB_DISPATCH_DTYPE(out_dtype, OT, [&]() -> int {
      const long long rows = (long long)T * H;
      if ((rows + 3) / 4 > 0x7fffffffLL) return gb::fail(GB_UNSUPPORTED, "delta_out: %d tokens of %d heads", T, H);
      auto kernel = vdim <= 32 ? delta_out_kernel<1, WT, OT> : vdim <= 64 ? delta_out_kernel<2, WT, OT> : vdim <= 128 ? delta_out_kernel<4, WT, OT>
                  : vdim <= 256 ? delta_out_kernel<8, WT, OT> : delta_out_any_kernel<WT, OT>;
      return gb::check_pdl_launch(gb::launch_pdl(kernel, dim3((unsigned)((rows + 3) / 4)), dim3(128), 0, stream, dim3(1, 1, 1), o,
                                                 second, P2, gate_off, (const WT*)w, eps, (OT*)out, H, vdim, silu_gate,
                                                 w_per_head, rows),
                                  "delta_out");
    });
  });
}

// One token per request (row t of the batch is request t). Takes vdim <= 256.
GB_EXPORT int gb_delta_decode(const float* proj, int P, const float* second, int P2, const void* conv_w, int w_dtype,
                              int taps, const float* conv_state, long long conv_stride, const void* a_log,
                              const void* dt_bias, const void* norm_w, float eps, const int32_t* slots, float* state,
                              long long state_stride, int R, int H, int G, int dim, int vdim, void* out, int out_dtype,
                              int per_head, int gate_off, int silu_gate, cudaStream_t stream) {
  if (R <= 0) return GB_OK;
  int rc = check_sizes("delta_decode", H, G, dim, vdim, taps);
  if (rc != GB_OK) return rc;
  if (vdim > 256) return gb::fail(GB_UNSUPPORTED, "delta_decode: %d value channels per head (at most 256)", vdim);
  const int threads = (vdim + 31) / 32 * 32;
  const size_t smem = (size_t)(3 * dim + 32 + vdim) * sizeof(float);
  return GB_DISPATCH_DTYPE(w_dtype, WT, [&]() -> int {
    return GB_DISPATCH_DTYPE(out_dtype, OT, [&]() -> int {
      return by_dim(dim, "delta_decode", [&](auto maxd) -> int {
        return gb::check_pdl_launch(
            gb::launch_pdl(delta_decode_kernel<decltype(maxd)::value, WT, OT>, dim3(H, R), dim3(threads), smem, stream,
                           dim3(1, 1, 1), proj, P, second, P2, (const WT*)conv_w, taps, conv_state, conv_stride,
                           (const WT*)a_log, (const WT*)dt_bias, (const WT*)norm_w, eps, slots, state, state_stride, H, G,
                           dim, vdim, (OT*)out, per_head, gate_off, silu_gate),
            "delta_decode");
      });
    });
  });
}
