// Shared device/host helpers for the difb200 kernels (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <utility>

namespace difb200 {

// Status codes are numerically identical to dif_backend_status of the reference plugin
// ABI (reference include/dif/backend/abi.h:22-30), so they pass through unchanged.
enum Status : int {
  kOk = 0,
  kInvalidArgument = 1,
  kUnsupported = 2,
  kOutOfMemory = 3,
  kCompileError = 4,
  kExecutionError = 5,
  kInternalError = 6,
};

// Thread-local text of the last failure, returned by difb200_last_error().
void set_last_error(const std::string &text);
int fail(int status, const std::string &text);
int check_cuda(cudaError_t code, const char *what);
// check_cuda for the status of a kernel launch; counts the launches of this process (launch_count).
int launched(cudaError_t code, const char *what);
unsigned long long launch_count();
int sm_count();

// One-time set-up that is per device, not per process (function attributes and occupancy
// figures belong to a context): `init` runs the first time `key` is seen with `device` and its
// result value is cached; a failing `init` is not cached. Thread-safe.
int per_device_once(const void *key, int device, int (*init)(void *arg, int *value), void *arg, int *value);
int current_device_once(const void *key, int (*init)(void *arg, int *value), void *arg, int *value);

// Blocks of `kernel` that are resident at once on one SM of the current device with this block size
// and dynamic shared memory; opts the kernel in to that much shared memory the first time. The
// answer is a property of the device and is looked up once per (kernel, device, block, bytes).
int resident_blocks(const void *kernel, int threads, size_t dynamic_smem, int *blocks);

// Device-side status words written by kernels whose bounded waits ran out. Index 0 is a
// sticky flag, 1..3 describe where (kernel id, role, iteration).
struct DeviceStatus {
  unsigned int flag;
  unsigned int kernel;
  unsigned int role;
  unsigned int detail;
};
// Limit of the kernels' bounded waits in nanoseconds (default 1.5 s), read at every launch.
unsigned long long wait_limit_ns();
void set_wait_limit_ns(unsigned long long ns); // 0 restores the default
// Test aid for the give-up path: the next LinearInt8Scaled launch leaves out the loads of one
// k-block. take_...() returns that k-block (0xffffffff = none) and disarms.
void withhold_next_gemm_load(uint32_t k_block);
uint32_t take_withheld_gemm_load();
bool gemm_load_is_withheld();
// The same for the quantiser of rows that are rotated one ahead of their maximum: a CTA of the next such launch waits for one
// announcement more of a row than its warps make, and the launch's waits have this limit. take_...() returns it (0 = not armed) and disarms.
void withhold_next_row_maximum(unsigned long long limit_ns);
unsigned long long take_withheld_row_maximum();
// Device memory for one call: allocated and freed in the order of the call's stream, so that neither
// another stream nor another thread can hold the same bytes meanwhile (also under stream capture, where the two become
// nodes of the graph). It comes from a pool of this library that keeps at most 4 MB per device across
// synchronisations. The consumer is launched on the same stream before the object goes.
class StreamScratch {
public:
  explicit StreamScratch(cudaStream_t stream) : stream_(stream) {}
  ~StreamScratch();
  StreamScratch(const StreamScratch &) = delete;
  StreamScratch &operator=(const StreamScratch &) = delete;
  int allocate(size_t bytes, const char *what); // once per object
  void *get() const { return data_; }

private:
  cudaStream_t stream_;
  void *data_ = nullptr;
};
DeviceStatus *device_status_words();      // per device, part of the library's image
int poll_device_status(const char *what); // copies back, clears, maps to kExecutionError

#ifdef __CUDACC__

// Division by a number that a launch fixes, of what is below 2^31: with 2^s the least power of two that is not below the
// divisor and mul = ceil(2^(31 + s) / by), mul * by exceeds 2^(31 + s) by e < 2^s, so n * e < 2^(31 + s) and the quotient
// of 2 n * mul and 2^(32 + s) is that of n and by.
struct Divisor {
  uint32_t by, mul, shift;
  __device__ __forceinline__ uint32_t quotient(uint32_t n) const { return __umulhi(2u * n, mul) >> shift; }
};
inline Divisor divisor(uint64_t by) { // 1 .. 2^31 - 1
  Divisor d{(uint32_t)by, 0, 0};
  while ((1ull << d.shift) < by)
    ++d.shift;
  d.mul = (uint32_t)(((1ull << (31 + d.shift)) + by - 1) / by);
  return d;
}

// ---- programmatic dependent launch ----
// A kernel launched with dependent_launch() may start while the one in front of it on the stream still runs: as soon as
// all CTAs of that one have called grid_dependents_launch() (or ended) and there is room. Its set-up runs then; what
// the kernel in front wrote is read behind grid_dependency_wait(), which every thread passes that touches global
// memory, and through loads that the compiler cannot move up: load_produced, TMA, or addresses that the wait is a part of
// (grid_dependency_wait_zero; the assembler keeps coherent loads behind the wait by itself). None of them is non-coherent
// (__ldg): that path is for memory that nobody writes while the kernel lives, and this one lives while the one in front
// writes. A kernel that lets dependents start waits first: when a kernel starts, the one two in front is complete.
// Two reads are not behind such a wait. Both are of what a kernel further in front wrote, and both hold only because
// the kernel in between waited before it let anything start (then that kernel is complete):
// * the first weights of a GEMM, requested ahead in w8a8_linear, whose quantiser is the kernel in between;
// * the operands of the attention's split launch: the unsplit one waits for their kernel, then fences, then lets it start.
// Launched plainly, a kernel starts 1 to 2.5 us after the end of the one in front; ahead, with a wait as the first thing
// it does, within half of one, whether or not that one says that dependents may start (calls of 2 x 3072 x 3072, one behind the
// other: 8.2 us, 5.9, and 5.8 where it says so at its start or its end). So it says so only where the next one has work to do
// meanwhile: CTAs that only wait would gather on the SMs that happen to be free.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The wait and a zero behind it: addresses of loads that could otherwise be moved in front of the wait (load_global) contain it.
__device__ __forceinline__ uint64_t grid_dependency_wait_zero() {
  uint64_t zero;
  asm volatile("griddepcontrol.wait;\nmov.u64 %0, 0;" : "=l"(zero)::"memory");
  return zero;
}
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ float load_produced(const float *p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t load_produced(const uint16_t *p) {
  uint16_t v;
  asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
// What __ldg is to the compiler, a value that depends on the address alone, by the coherent path. Like __ldg it is not for memory that
// this kernel writes before.
__device__ __forceinline__ uint4 load_global(const uint4 *p) {
  uint4 v;
  asm("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 load_global(const float4 *p) {
  float4 v;
  asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 load_global(const float2 *p) {
  float2 v;
  asm("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float load_global(const float *p) {
  float v;
  asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t load_global(const uint16_t *p) {
  uint16_t v;
  asm("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 load_produced(const uint4 *p) {
  uint4 v;
  asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// 16 bytes that are read once. The second form is for what no kernel that may still run has written.
__device__ __forceinline__ uint4 load_produced_once(const void *p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 load_streamed(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
inline cudaLaunchAttribute dependent_launch() {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  return attr;
}
// Launches a kernel that begins with its wait.
template <class... P, class... A>
int launch_ahead(const char *what, void (*kernel)(P...), uint64_t grid, int threads, size_t smem, cudaStream_t stream, A &&...args) {
  cudaLaunchConfig_t config{};
  config.gridDim = dim3((unsigned)grid);
  config.blockDim = dim3((unsigned)threads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attr = dependent_launch();
  config.attrs = &attr;
  config.numAttrs = 1;
  return launched(cudaLaunchKernelEx(&config, kernel, std::forward<A>(args)...), what);
}

__device__ __forceinline__ float bf16_bits_to_f32(uint32_t bits16) {
  return __uint_as_float(bits16 << 16);
}
// Round-to-nearest-even on the raw fp32 bits, the reference's bf16 store
// (reference src/runtime/scalar.cpp:18-22). The NaN of this GPU's arithmetic, 0x7fffffff, would overflow to -0 there, where
// that of a CPU (0x7fc00000, 0xffc00000) stays a NaN: the minimum keeps it one (0x7fff) and changes nothing else.
__device__ __forceinline__ uint32_t number_to_bf16_bits(uint32_t b) {
  return ((b + 0x7fffu + ((b >> 16) & 1u)) >> 16) & 0xffffu;
}
__device__ __forceinline__ uint32_t f32_to_bf16_bits(float v) {
  return number_to_bf16_bits((uint32_t)min(__float_as_int(v), 0x7fff7fff));
}
__device__ __forceinline__ float round_bf16(float v) {
  return __uint_as_float(f32_to_bf16_bits(v) << 16);
}
// The same of what is never NaN (a row scale).
__device__ __forceinline__ float round_bf16_number(float v) {
  return __uint_as_float(number_to_bf16_bits(__float_as_uint(v)) << 16);
}

// ---- packed fp32x2 arithmetic (two independent fp32 lanes per 64-bit register) ----
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

#endif // __CUDACC__

} // namespace difb200
