// out[M,N] (+)= a[M,K] * w[N,K]^T on the ordinary (non-tensor) cores, with true
// 32-bit multiply-adds: the matrix product of the 32-bit path, and the check
// beside the tensor-core kernels. garuda/src/simd/mod.rs:96-129 (`matmul`: each
// output is the dot of one matrix row with one input vector, :13-16).
//
// Every output element is a sum over k = 0..K-1 in an order that N and K alone decide, whatever M is, so a
// token's result does not depend on the rest of the batch: in ascending order, and in the tiled kernel (32-bit operands whose
// rows start on 16 bytes) the even and the odd k by themselves, of up to eight parts of K, added in the order of the parts.
#include <cooperative_groups.h>

#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;  // 256 threads, 4x4 outputs each

template <typename IT, typename OT, bool ACCUMULATE>
__global__ void __launch_bounds__(256)
gemm_simple_kernel(const IT* __restrict__ a, const IT* __restrict__ w, OT* __restrict__ out, int M, int N,
                   int K, float alpha) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tm = (tid / 16) * TM, tn = (tid % 16) * TN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 rows x 16 columns per operand: 1024 elements, 4 per thread
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * 256;
      const int r = e / BK, c = e % BK;
      const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? gb::to_float<IT>(a[(size_t)gm * K + gk]) : 0.f;
      Ws[c][r] = (gn < N && gk < K) ? gb::to_float<IT>(w[(size_t)gn * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float av[TM], wv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = As[k][tm + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) wv[j] = Ws[k][tn + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + tm + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tn + j;
      if (gn >= N) continue;
      OT* o = out + (size_t)gm * N + gn;
      if (ACCUMULATE) *o = gb::from_float<OT>(fmaf(alpha, acc[i][j], gb::to_float<OT>(*o)));
      else *o = gb::from_float<OT>(acc[i][j]);
    }
  }
}

// ---- 32-bit operands: tiles of BM x 128, BM = 8 to 64 by the number of rows ------------------------
//
// What bounds it: the multiply-add rate for many rows (117 a clock and SM measured, 67 TFLOP/s), the stream of weights for few. A
// number read from shared memory costs a lane's 4 bytes of its 128 a clock, half of that where neighbouring lanes read
// the same (an A row), so a thread's 8 x 8 outputs take 12 clocks of shared memory for 16 of multiply-adds, and at 8 rows a weight is read by
// two lanes only. Operands stay as they lie in memory, four k side by side (16-byte copies, 16-byte
// reads; rows 36 floats apart fall into different banks). The CTAs of a cluster split K where N has too few tiles to fill the GPU,
// by a rule on N and K alone, exchange their tiles through distributed shared memory and add them in order.
// Measured (B200): [500, 2048] x [11264, 2048]^T 815 us with 64 x 64 tiles and single reads, 588 in this shape with one multiply-add an
// instruction (three operands of their own each: 55 TFLOP/s at most where two at once reach 67), 554 now (42 TFLOP/s);
// [2, 2048] x [32000, 2048]^T 360 -> 63 us (4.1 TB/s).
constexpr int TBN = 128, TBK = 32, TLD = TBK + 4, TOUT = TBN + 4;
constexpr int TILE_THREADS = 128;

__device__ __forceinline__ void copy_16(float* smem, const float* gmem, bool valid) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}

// two 32-bit multiply-adds in one instruction, on numbers that lie side by side
using pair_t = unsigned long long;
struct __align__(16) pair2_t { pair_t a, b; };
__device__ __forceinline__ void fma2(pair_t& d, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ float sum_of_pair(pair_t p) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
  return lo + hi;
}

// A warp has BM rows and 32 of the columns; a thread TM rows (RG apart) and TN columns (CL apart).
template <int TM, int TN, int RG, int STAGES, typename OT, bool ACCUMULATE>
__global__ void __launch_bounds__(TILE_THREADS)
gemm_tile_kernel(const float* __restrict__ a, const float* __restrict__ w, OT* __restrict__ out, int M, int N, int K, float alpha) {
  constexpr int BM = TM * RG, CL = 32 / RG;
  static_assert(TN * CL * (TILE_THREADS / 32) == TBN, "the warps cover the tile's columns");
  constexpr int STAGE = (BM + TBN) * TLD;
  extern __shared__ __align__(16) float sh[];          // STAGES stages; then the tile [BM][TOUT]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rg = lane / CL, cl = lane % CL;
  const int n0 = blockIdx.x * TBN, m0 = blockIdx.y * BM, split = gridDim.z, rank = blockIdx.z;
  const int blocks = (K + TBK - 1) / TBK;
  const int first = (int)((long long)blocks * rank / split), last = (int)((long long)blocks * (rank + 1) / split);
  auto load = [&](int block) {
    if (block < last) {
      float* st = sh + (block - first) % STAGES * STAGE;
      const int k0 = block * TBK;
#pragma unroll
      for (int i = tid; i < (BM + TBN) * (TBK / 4); i += TILE_THREADS) {
        const int row = i / (TBK / 4), k = k0 + i % (TBK / 4) * 4;
        const bool is_a = row < BM;
        const int at = is_a ? m0 + row : n0 + row - BM;
        const bool ok = k < K && at < (is_a ? M : N);
        copy_16(st + row * TLD + i % (TBK / 4) * 4, (is_a ? a : w) + (ok ? (size_t)at * K + k : 0), ok);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  pair_t acc[TM][TN];                                  // the sums over even k and over odd k
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load(first + s);
  for (int block = first; block < last; ++block) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                   // this block has landed; everyone is done with the one in front
    load(block + STAGES - 1);
    const float* as = sh + (block - first) % STAGES * STAGE + rg * TLD;
    const float* ws = sh + (block - first) % STAGES * STAGE + (BM + warp * (TBN / 4) + cl) * TLD;
#pragma unroll
    for (int kk = 0; kk < TBK; kk += 4) {
      pair2_t b[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const pair2_t*>(ws + j * CL * TLD + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const pair2_t x = *reinterpret_cast<const pair2_t*>(as + i * RG * TLD + kk);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], x.a, b[j].a);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], x.b, b[j].b);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sh[(rg + i * RG) * TOUT + warp * (TBN / 4) + cl + j * CL] = sum_of_pair(acc[i][j]);
  namespace cg = cooperative_groups;
  if (split > 1) cg::this_cluster().sync();
  else __syncthreads();
  // the ranks share the tile's rows out; the CTAs' sums are added in the order of their parts of K
  for (int i = rank * TILE_THREADS + tid; i < BM * (TBN / 4); i += split * TILE_THREADS) {
    const int row = i / (TBN / 4), col = i % (TBN / 4) * 4;
    if (m0 + row >= M) continue;
    float* mine = sh + row * TOUT + col;
    float4 sum;
    if (split > 1) {
      float4 part[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < split) part[r] = *reinterpret_cast<const float4*>(cg::this_cluster().map_shared_rank(mine, r));
      sum = part[0];
#pragma unroll
      for (int r = 1; r < 8; ++r)
        if (r < split) sum.x += part[r].x, sum.y += part[r].y, sum.z += part[r].z, sum.w += part[r].w;
    } else {
      sum = *reinterpret_cast<const float4*>(mine);
    }
    const float v[4] = {sum.x, sum.y, sum.z, sum.w};
    OT* o = out + (size_t)(m0 + row) * N + n0 + col;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (n0 + col + e < N) o[e] = gb::from_float<OT>(ACCUMULATE ? fmaf(alpha, v[e], gb::to_float<OT>(o[e])) : v[e]);
  }
  if (split > 1) cg::this_cluster().sync();            // a rank's tile stays until all have read it
}

// Into how many parts K is cut: what makes about as many CTAs of one row of tiles as there are SMs (a quarter more), a part no shorter
// than 128. Of N and K alone (see the top).
int parts_of_k(int N, int K) {
  const int tiles = (N + TBN - 1) / TBN;
  int parts = 185 / tiles;
  if (parts > K / 128) parts = K / 128;
  return parts < 1 ? 1 : parts > 8 ? 8 : parts;
}

template <int TM, int TN, int RG, int STAGES, typename OT, bool ACCUMULATE>
int launch_tile(const float* a, const float* w, OT* out, int M, int N, int K, float alpha, cudaStream_t stream) {
  constexpr int BM = TM * RG;
  constexpr size_t smem = (size_t)STAGES * (BM + TBN) * TLD * sizeof(float);
  static_assert(smem >= (size_t)BM * TOUT * sizeof(float), "the finished tile takes the stages' place");
  auto kernel = gemm_tile_kernel<TM, TN, RG, STAGES, OT, ACCUMULATE>;
  static gb::OncePerDevice configured;
  if (configured.needed()) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "gemm: %s", cudaGetErrorString(e));
    configured.done();
  }
  const int parts = parts_of_k(N, K);
  const cudaError_t e = gb::launch_after(kernel, dim3((N + TBN - 1) / TBN, (M + BM - 1) / BM, parts), dim3(TILE_THREADS), smem, stream,
                                         dim3(1, 1, parts), a, w, out, M, N, K, alpha);
  if (e != cudaSuccess) return gb::fail(GB_CUDA_ERROR, "gemm: %s", cudaGetErrorString(e));
  return gb::check_launch("gemm_tile");
}

// A tile's rows change no number, so M may choose them: the fewest that hold all of M, or whose tiles all find an SM of their own. (64 rows
// for every M above 32 left small products to a few slow tiles: [128, 128] x [256, 128]^T 12.4 us, in the 64 x 64 tiles of the other kernel 10.4,
// now 6.3; [2048, 64] x [64, 64]^T 8.3, 6.3, 3.6.)
template <typename OT, bool ACCUMULATE>
int gemm_tiled(const float* a, const float* w, OT* out, int M, int N, int K, float alpha, cudaStream_t stream) {
  const long long columns = (long long)((N + TBN - 1) / TBN) * parts_of_k(N, K);
  auto suits = [&](int rows) { return M <= rows || columns * ((M + rows - 1) / rows) <= gb::sm_count(); };
  if (M <= 8) return launch_tile<4, 2, 2, 5, OT, ACCUMULATE>(a, w, out, M, N, K, alpha, stream);
  if (suits(16)) return launch_tile<4, 4, 4, 5, OT, ACCUMULATE>(a, w, out, M, N, K, alpha, stream);
  if (suits(32)) return launch_tile<8, 4, 4, 3, OT, ACCUMULATE>(a, w, out, M, N, K, alpha, stream);
  return launch_tile<8, 8, 8, 3, OT, ACCUMULATE>(a, w, out, M, N, K, alpha, stream);
}

}  // namespace

// in_dtype: dtype of a and w; out_dtype: dtype of out. accumulate: out += alpha * product
// (out must then be 32-bit: it is the residual stream; alpha is a model's residual multiplier).
GB_EXPORT int gb_gemm_simple(const void* a, const void* w, void* out, int M, int N, int K, int in_dtype,
                             int out_dtype, int accumulate, float alpha, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return GB_OK;
  if (K <= 0) return gb::fail(GB_BAD_ARGUMENT, "gemm: K = %d", K);
  if (accumulate && out_dtype != GB_F32)
    return gb::fail(GB_BAD_ARGUMENT, "gemm: accumulation needs a 32-bit output");
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  // the tiled kernel copies 16 bytes at a time; with a single block of 32 channels it gains nothing (up to 1.5 times the other's 4 us)
  if (in_dtype == GB_F32 && K % 4 == 0 && K > TBK && (((uintptr_t)a | (uintptr_t)w) & 15) == 0) {
    return GB_DISPATCH_DTYPE(out_dtype, OT, [&]() -> int {
      return accumulate ? gemm_tiled<OT, true>((const float*)a, (const float*)w, (OT*)out, M, N, K, alpha, stream)
                        : gemm_tiled<OT, false>((const float*)a, (const float*)w, (OT*)out, M, N, K, alpha, stream);
    });
  }
  return GB_DISPATCH_DTYPE(in_dtype, IT, [&]() -> int {
    return GB_DISPATCH_DTYPE(out_dtype, OT, [&]() -> int {
      if (accumulate)
        gemm_simple_kernel<IT, OT, true><<<grid, 256, 0, stream>>>((const IT*)a, (const IT*)w, (OT*)out, M, N, K, alpha);
      else
        gemm_simple_kernel<IT, OT, false><<<grid, 256, 0, stream>>>((const IT*)a, (const IT*)w, (OT*)out, M, N, K, alpha);
      return gb::check_launch("gemm_simple");
    });
  });
}
