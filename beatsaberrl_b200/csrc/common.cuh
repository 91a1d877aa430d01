// Shared device/host helpers for the policy-forward kernels (sm_100a only).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <mutex>

#include "../../include/bsrl.h"

namespace bsrl {

constexpr int kT = BSRL_N_TOKENS;      // 29 tokens per env
constexpr int kLead = BSRL_N_LEAD;     // 5 lead tokens
constexpr int kSlots = BSRL_N_SLOTS;   // 24 entity slots
constexpr int kObs = BSRL_OBS_DIM;     // 630 obs lanes
constexpr int kActHeads = BSRL_N_ACT_HEADS;
constexpr float kMaskBias = 16384.0f;  // additive key mask magnitude
constexpr float kMaskedLogit = -1e9f;  // fill of lanes past a head's gear count

// Quotient and remainder of a row or element index (0 <= i) by a small positive divisor.  64-bit integer
// division is a long software routine on the GPU (~150 cycles per call where a thread needs it before it can do
// anything else); indices that fit 32 bits -- all of them at the sizes these kernels see -- take the 32-bit
// unsigned division instead.
__host__ __device__ __forceinline__ int64_t div_index(int64_t i, int d, int* rem) {
  if (!((uint64_t)i >> 32)) {
    const uint32_t q = (uint32_t)i / (uint32_t)d;
    *rem = (int)((uint32_t)i - q * (uint32_t)d);
    return (int64_t)q;
  }
  *rem = (int)(i % d);
  return i / d;
}

// Row remapping of a (rows, ld) matrix: logical row r lives at physical row
// (r / group) * stride + first + (r % group).  Identity: group = INT_MAX, stride = 0, first = 0.
struct PlainMap {
  int group;
  int stride;
  int first;
  __host__ __device__ inline int64_t operator()(int64_t r) const {
    if (r < (int64_t)group) return (int64_t)first + r;      // identity maps and every first group: no division
    int rem;
    const int64_t q = div_index(r, group, &rem);
    return q * (int64_t)stride + first + rem;
  }
  // the same map as the plain formula, for cold paths of kernels whose code generation should not move
  __host__ __device__ inline int64_t plain(int64_t r) const {
    return (r / group) * (int64_t)stride + first + (r % group);
  }
  bool dense() const { return group == 0x7fffffff && stride == 0 && first == 0; }
};
// Packed token rows (rows.cu): the groups start at start[r / group] instead of at multiples of stride.  Kernels that never
// see these take the plain part: their parameters' place is latency of small launches.
struct RowMap : PlainMap {
  const int* start = nullptr;
  RowMap() = default;
  __host__ __device__ RowMap(int g, int s, int f, const int* t = nullptr) : PlainMap{g, s, f}, start(t) {}
  __device__ inline int64_t operator()(int64_t r) const {
    if (!start) return PlainMap::operator()(r);
    int rem;
    const int64_t q = div_index(r, group, &rem);
    return (int64_t)start[q] + first + rem;
  }
  bool dense() const { return PlainMap::dense() && !start; }
};
inline RowMap identity_map() { return RowMap{0x7fffffff, 0, 0}; }

// thread-local error message (host)
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);

#define BSRL_CUDA_OK(expr)                                   \
  do {                                                       \
    cudaError_t e__ = (expr);                                \
    if (e__ != cudaSuccess) return ::bsrl::cuda_fail(e__, #expr); \
  } while (0)

#define BSRL_LAUNCH_OK(what)                                 \
  do {                                                       \
    cudaError_t e__ = cudaGetLastError();                    \
    if (e__ != cudaSuccess) return ::bsrl::cuda_fail(e__, what); \
  } while (0)

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

int sm_count();  // multiprocessors of the current device (cached per device)

// One-time set-up per device (raising a kernel's dynamic shared-memory limit, resolving a device
// symbol): run(what, fn) calls fn() -> cudaError_t once for the CURRENT device, whichever host
// thread gets there first, and returns BSRL_OK or the failure of that first run.  The cached result
// belongs to the device's primary context: it does not survive cudaDeviceReset.
constexpr int kMaxDevices = 64;
class DeviceOnce {
 public:
  template <typename Fn>
  int run(const char* what, Fn&& fn) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) {
      set_error("%s: device ordinal %d not supported (at most %d devices)", what, dev, kMaxDevices);
      return BSRL_ERR_UNSUPPORTED;
    }
    std::call_once(flag_[dev], [&] { err_[dev] = fn(); });
    if (err_[dev] != cudaSuccess) return cuda_fail(err_[dev], what);
    return BSRL_OK;
  }

 private:
  std::once_flag flag_[kMaxDevices];
  cudaError_t err_[kMaxDevices] = {};
};

// Kernel launches.  Inside a sequence (PdlScope, after pdl_enable()) a launch is programmatic: the kernel may start while
// its predecessor still runs, does what needs nothing of it (barriers, TMEM, weight loads) and waits in pdl_wait()
// until every earlier kernel has completed and its writes are visible; outside of one it is an ordinary launch and
// pdl_wait() returns at once.  Every kernel launched this way calls pdl_wait() before it touches anything an earlier
// kernel of the sequence wrote or reads, and pdl_trigger() only after it: a successor's early part therefore runs when
// at most ONE predecessor is unfinished, so reading the weights there is safe as long as no kernel of the sequence
// writes them (the pack kernels run outside of sequences).
extern thread_local bool g_pdl;
inline void pdl_enable() { g_pdl = true; }
struct PdlScope {
  ~PdlScope() { g_pdl = false; }
};
template <int CLUSTER = 1, typename... P, typename... A>
inline void launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (g_pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (CLUSTER > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = CLUSTER;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);     // BSRL_LAUNCH_OK follows every launch
}

// ----------------------------------------------------------------------------- device
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// the first statement of a kernel with nothing to do ahead of its predecessor
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_trigger();
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool pred) {
  int n = pred ? 16 : 0;  // src-size 0 => zero fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x2(uint32_t& r0, uint32_t& r1, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

// D(16x8, f32) += A(16x16, f16 row) * B(16x8, f16 col)
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                        uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Two fp32 operations per instruction (an even / odd register pair): the epilogues that work on every element of a wide
// activation are bound by the instructions they issue.
__device__ __forceinline__ uint64_t f2_make(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_split(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// erf-based GELU, 0.5 x (1 + erf(x / sqrt 2)): torch.nn.GELU() with its default approximate='none'.
// x Phi(x) = max(x, 0) - |x| Phi(-|x|) with Phi(-a) = 2^q(a), q a polynomial: minimax fits (linear programmes over Chebyshev
// nodes, this file's own) of log2 Phi(-a), whose negative leading coefficients take q to minus infinity past the fit.  One
// special-function instruction per element.
// Results that are rounded to fp16: degree 8, fitted to [0, 6.2] for an absolute error below 1e-7 x and, down to x = -4, a
// relative error of the negative branch below 2e-5.  Past -4 that grows (2.5e-4 at -4.5, 2e-3 at -5, 3.5e-2 at -6, all of the
// result past -8), which is 1.2e-8 at most there: a fifth of fp16's smallest step.  FMAs two elements at a time.
// fp32 results: degree 12, fitted to [0, 12.9], where the result itself runs out of fp32: relative error of the negative branch
// below 6e-7 to -2, 5e-6 to -4, 4e-5 to -6, 3e-4 to -8, 1e-3 to -10, 9e-3 to -12.9.
// In fp32 against float64 over [-12.9, 12.9], degree 8 / degree 12 / the rational-exponential form 7.1.26 of Abramowitz & Stegun
// with a reciprocal and an exponential: largest error 2.4e-7 / 2.4e-7 / 3.3e-7, rms 4.1e-8 / 4.0e-8 / 7.3e-8, relative on [-4, 0)
// 1.1e-5 / 5.0e-6 / 4.7e-4, on [-8, -4) 0.72 / 2.9e-4 / 1.0e-2; of results rounded to fp16, 0.3 % / - / 2.8 % differ from the
// rounded exact value.  Degree 8 against 7.1.26: 65,536 environments of 33 tokens at d 256 18.98 -> 17.79 ms per forward; 4,095
// of 65 at d 512 (the FFN-up's epilogue took longer than its MMAs): 14.08 -> 12.38 ms before the power cap sets in, 14.52 ->
// 13.71 in a loop.
__device__ constexpr float kGeluQ[9] = {-9.99999744e-01f, -1.15111655e+00f, -4.59124456e-01f, -5.27288577e-02f, 7.37600707e-03f,
                                        -3.61215035e-04f, -9.85613870e-05f, 2.18674498e-05f, -1.43885577e-06f};
__device__ constexpr float kGeluQ32[13] = {-1.00000000e+00f, -1.15110564e+00f, -4.59209889e-01f, -5.24704345e-02f, 6.98015373e-03f,
                                           -1.46172151e-05f, -2.82148336e-04f, 8.17496766e-05f, -1.33107760e-05f, 1.37389475e-06f,
                                           -8.84585063e-08f, 3.23252669e-09f, -5.10666856e-11f};
__device__ __forceinline__ float gelu_ex2(float q) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(q));
  return e;
}
template <int N>
__device__ __forceinline__ float gelu_of(float x, const float (&c)[N]) {
  const float a = fabsf(x);
  float q = c[N - 1];
#pragma unroll
  for (int i = N - 2; i >= 0; --i) q = fmaf(q, a, c[i]);
  return fmaf(-a, gelu_ex2(q), fmaxf(x, 0.f));
}
__device__ __forceinline__ float gelu_f16(float x) { return gelu_of(x, kGeluQ); }      // rounded to fp16 by the caller
__device__ __forceinline__ float gelu_f32(float x) { return gelu_of(x, kGeluQ32); }
// the same, two at a time (bit for bit)
template <bool F32>
__device__ __forceinline__ void gelu2(float& x0, float& x1) {
  constexpr int N = F32 ? 13 : 9;
  const uint64_t a = f2_make(fabsf(x0), fabsf(x1));
  auto c = [](int i) { return F32 ? kGeluQ32[i] : kGeluQ[i]; };
  uint64_t q = f2_make(c(N - 1), c(N - 1));
#pragma unroll
  for (int i = N - 2; i >= 0; --i) q = f2_fma(q, a, f2_make(c(i), c(i)));
  float q0, q1;
  f2_split(q, q0, q1);
  f2_split(f2_fma(f2_make(-fabsf(x0), -fabsf(x1)), f2_make(gelu_ex2(q0), gelu_ex2(q1)), f2_make(fmaxf(x0, 0.f), fmaxf(x1, 0.f))), x0, x1);
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

}  // namespace bsrl
