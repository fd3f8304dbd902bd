// Shared device/host helpers for the NSA sm_100a kernels.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>
#include <math.h>

#include "../../include/nsa_b200.h"

namespace nsa {

// Records a message that nsa_last_error() returns and yields `code`.
int fail(int code, const char* fmt, ...);

#define NSA_REQUIRE(cond, code, ...)                 \
  do {                                               \
    if (!(cond)) return ::nsa::fail((code), __VA_ARGS__); \
  } while (0)

#define NSA_CUDA_OK(expr)                                                         \
  do {                                                                            \
    cudaError_t e__ = (expr);                                                     \
    if (e__ != cudaSuccess)                                                       \
      return ::nsa::fail(NSA_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e__)); \
  } while (0)

static inline int launch_status(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(NSA_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(e));
  return NSA_OK;
}

// ---------------------------------------------------------------- programmatic dependent launch
// A kernel launched through launch_pdl may become resident while the kernel before it in the stream is still running,
// which takes the launch latency and its own set-up off the path between the two.  It must execute grid_dep_wait()
// before its first access to global memory (reads, and writes to memory an earlier kernel may still read): that waits
// for the whole kernel before it, and -- because every kernel of the chain waits the same way -- for all before that.
// grid_dep_launch() lets the next kernel of the stream become resident early; what it waits for does not change.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static inline int launch_pdl(const char* what, void (*kernel)(KArgs...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
  if (e != cudaSuccess) return fail(NSA_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(e));
  return NSA_OK;
}

// One tensor of a pooling launch: window means of x [slabs, T, D] into out [slabs, n_out, D] (pool_select.cu).
struct PoolJob {
  const void* x;
  void* out;
  int T, block, stride, n_out, slabs;
  float dq;            // fp8 only: factor of the dequantisation
  unsigned block0;     // filled in by the launcher
};

// Backward of the whole forward, fp16 storage: gate * P, which has no gate-independent size, is held as 2^14 times itself.  It is
// at most 1, so nothing overflows, and values down to 4e-9 keep all 11 bits (unscaled: 6e-5, which gate logits of -6
// over a few thousand keys fall below, and no scaling of the loss can reach).  bf16 has the exponents of fp32.
constexpr float kGatedPExp = 14.f, kGatedPInv = 1.f / 16384.f;

// ---------------------------------------------------------------- dtype traits
template <typename T> struct Elem;
template <> struct Elem<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  static __device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float x) { return __float2bfloat16_rn(x); }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  }
};
template <> struct Elem<__half> {
  using T2 = __half2;
  static __device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half from_f(float x) { return __float2half_rn(x); }
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  static __device__ __forceinline__ float2 unpack(uint32_t u) {
    return __half22float2(*reinterpret_cast<__half2*>(&u));
  }
};

// fp8 byte -> fp32 (exact).  fmt: NSA_FP8_E4M3 / NSA_FP8_E5M2
__device__ __forceinline__ float fp8_to_f(uint8_t b, int fmt) {
  __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)b, fmt == NSA_FP8_E5M2 ? __NV_E5M2 : __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// 16-byte async copy; src_bytes == 0 zero-fills the destination.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
// D(16x8,f32) += A(16x16) * B(16x8)
template <typename T>
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma16816<__half>(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared-memory tile of rows x D 16-bit elements, 16-byte chunks XOR-swizzled so that
// ldmatrix (8 rows, one chunk column) and row-wise cp.async are both conflict-free.
template <int D>
__device__ __forceinline__ uint32_t tile_off(int row, int chunk) {
  constexpr int CH = D / 8;                       // chunks per row
  if constexpr (CH >= 8) return (uint32_t)(row * (D * 2) + ((chunk ^ (row & 7)) << 4));
  else if constexpr (CH == 4) return (uint32_t)(row * (D * 2) + ((chunk ^ ((row >> 1) & 3)) << 4));
  else return (uint32_t)(row * (D * 2) + ((chunk ^ ((row >> 2) & 1)) << 4));
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

}  // namespace nsa
