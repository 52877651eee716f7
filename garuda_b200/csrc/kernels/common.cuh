// Shared by every kernel file: error reporting, dtype tags, conversions.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#define GB_EXPORT extern "C" __attribute__((visibility("default")))

// dtype tags of the C interface
enum GbDtype : int { GB_F32 = 0, GB_BF16 = 1 };

// Status codes returned by every entry point. 0 is success; the text of the
// last failure of the calling thread is available from gb_last_error().
enum GbStatus : int { GB_OK = 0, GB_BAD_ARGUMENT = 1, GB_CUDA_ERROR = 2, GB_UNSUPPORTED = 3 };

namespace gb {

inline char* error_buffer() {
  static thread_local char buf[512];
  return buf;
}

inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(error_buffer(), 512, fmt, ap);
  va_end(ap);
  return code;
}

inline int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(GB_CUDA_ERROR, "%s: %s", what, cudaGetErrorString(e));
  return GB_OK;
}

template <typename T>
__device__ __forceinline__ float to_float(T v);
template <>
__device__ __forceinline__ float to_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T from_float(float v);
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
// Two neighbouring values, each rounded as from_float rounds it, in one store; `to` is an even element of a row
// that starts on 8 bytes.
__device__ __forceinline__ void store_pair(float* to, float a, float b) { *reinterpret_cast<float2*>(to) = make_float2(a, b); }
__device__ __forceinline__ void store_pair(__nv_bfloat16* to, float a, float b) {
  *reinterpret_cast<__nv_bfloat162*>(to) = __nv_bfloat162(__float2bfloat16_rn(a), __float2bfloat16_rn(b));
}

// 1 / d and z / d, rounded, of a d from 1 to infinity (the denominators of sigmoid and SiLU), without a branch, so that a thread's many
// stand beside one another: Newton's step from the hardware's approximation, then Markstein's correction of the quotient ("Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990). The approximation is asked for at an eighth of d, where neither it nor
// its operand is subnormal; the steps are at d itself, so that a result which is subnormal is rounded once. `over` gives the division's bits for every d up to
// 2^126 and for all but five beyond (which are a last place off); `divide` gives them for every z over 1 + exp(-z) (small z meet d = 2),
// and for other z and d where z is at least 2^-100 and the result is normal.
__device__ __forceinline__ float over_first(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(0.125f * d));
  return 0.125f * r;
}
__device__ __forceinline__ float over(float d) {
  const float a = over_first(d);
  return d < INFINITY ? fmaf(a, fmaf(-d, a, 1.0f), a) : a;
}
__device__ __forceinline__ float divide(float z, float d) {
  const float a = over_first(d), r = fmaf(a, fmaf(-d, a, 1.0f), a), q = z * r;
  const float better = fmaf(fmaf(-q, d, z), r, q);
  return copysignf(d < INFINITY && fabsf(better) < INFINITY ? better : z * a, z);      // (a zero's sign is lost on the way)
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// A kernel attribute (the dynamic shared memory a kernel may use) belongs to a device: a flag that
// remembers "set" must be kept per device. `needed()` is true until `done()` has been called with
// the same device current. Not synchronised: two threads that make a kernel's first call on a
// device at the same moment both set the attribute, to the same value.
struct OncePerDevice {
  static constexpr int MAX_DEVICES = 64;
  bool set_[MAX_DEVICES] = {};
  static int device() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= MAX_DEVICES) return -1;
    return d;
  }
  bool needed() const {
    const int d = device();
    return d < 0 || !set_[d];
  }
  void done() {
    const int d = device();
    if (d >= 0) set_[d] = true;
  }
};

// SMs of the device that was current at the first call.
inline int sm_count() {
  static const int n = [] {
    int dev = 0, v = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

// ---- programmatic dependent launch ----------------------------------------
// A kernel launched with launch_pdl may start while the kernel before it in the
// stream is still running. It must call pdl_wait() before it reads anything that
// kernel wrote and before it writes anything that kernel may still read; what it
// does before that (setting up barriers, fetching weights) overlaps the tail of
// its predecessor. pdl_launch_dependents() lets the kernel after it start early
// in the same way. Both are no-ops for a kernel launched the ordinary way.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

inline bool pdl_enabled() {
  static const bool on = [] {
    const char* v = getenv("GARUDA_B200_PDL");
    return !(v && v[0] == '0');
  }();
  return on;
}

// Launch with the programmatic-serialization attribute, and as clusters of the given shape if it
// holds more than one CTA.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_with(bool early, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                               dim3 cluster, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attrs[2];
  int n = 0;
  if (early && pdl_enabled()) {
    attrs[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster.x * cluster.y * cluster.z > 1) {
    attrs[n].id = cudaLaunchAttributeClusterDimension;
    attrs[n].val.clusterDim.x = cluster.x;
    attrs[n].val.clusterDim.y = cluster.y;
    attrs[n].val.clusterDim.z = cluster.z;
    ++n;
  }
  cfg.attrs = attrs;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              dim3 cluster, Args... args) {
  return launch_with(true, kernel, grid, block, smem, stream, cluster, args...);
}

// The ordinary launch: the kernel starts when the one before it in the stream has finished. For a
// kernel of few, long-running blocks: started early, its blocks are placed while the predecessor's
// still hold the SMs (on whichever have room, it seems, several to an SM) and stay there for the
// kernel's whole time (the generalized delta rule's recurrence, 128 blocks over 2,048 tokens:
// 1.9 ms started early, 0.77 ms started after).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_after(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                dim3 cluster, Args... args) {
  return launch_with(false, kernel, grid, block, smem, stream, cluster, args...);
}

inline int check_pdl_launch(cudaError_t e, const char* what) {
  if (e != cudaSuccess) return fail(GB_CUDA_ERROR, "%s: %s", what, cudaGetErrorString(e));
  return check_launch(what);
}

}  // namespace gb

// One file of each library places this, so that the library exports the text
// of the calling thread's last failure.
#define GB_DEFINE_LAST_ERROR() \
  GB_EXPORT const char* gb_last_error() { return gb::error_buffer(); }

// Dispatch on a dtype tag: runs `body` with `T` bound to float or __nv_bfloat16.
#define GB_DISPATCH_DTYPE(tag, T, ...)                                   \
  [&]() -> int {                                                         \
    if ((tag) == GB_F32) { using T = float; return __VA_ARGS__(); }      \
    if ((tag) == GB_BF16) { using T = __nv_bfloat16; return __VA_ARGS__(); } \
    return gb::fail(GB_BAD_ARGUMENT, "unknown dtype tag %d", (int)(tag)); \
  }()
