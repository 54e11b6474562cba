// Shared host/device helpers for libhyperattn_b200 (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <atomic>

#include "hyperattn_b200.h"

namespace ha {

constexpr int TILE = 128;           // rows per attention tile (the reference's BLOCK_M = BLOCK_N)
constexpr int SPIN_LIMIT = 1 << 18;  // poll cap of every device-side wait (a legitimate wait is a few microseconds)
// ... and its time cap in SM clock cycles (about a second): one try_wait may itself suspend the thread for a
// hardware-chosen while, so a count of polls alone bounds nothing in practice (measured: minutes)
constexpr long long WAIT_CYCLES = 2000000000LL;

extern std::atomic<long long> g_launches;
void set_cuda_error(cudaError_t e, const char* where);

#define HA_CUDA_OK(expr, where)                                   \
  do {                                                            \
    cudaError_t _e = (expr);                                      \
    if (_e != cudaSuccess) {                                      \
      ::ha::set_cuda_error(_e, where);                            \
      return HA_ERR_CUDA;                                         \
    }                                                             \
  } while (0)

#define HA_LAUNCHED(where)                                        \
  do {                                                            \
    ::ha::g_launches.fetch_add(1, std::memory_order_relaxed);     \
    HA_CUDA_OK(cudaGetLastError(), where);                        \
  } while (0)

// Launch of a kernel that begins with chain_begin(): its CTAs may be placed while the last CTAs of the stream's previous kernel still run, and wait there
// for that kernel's end (programmatic stream serialization).  The launch and the first CTAs' start then lie under the tail of the kernel before.  Used
// where that is worth something and does no harm: the attention kernels (one CTA an SM), the sorts, merges and finishing passes behind
// them.  Kernels of several CTAs an SM in one wave are placed unevenly when SMs come free one by one (fp32 attention 122 -> 142 us), hash, delta and
// cast gained nothing.  The same library with and without the attribute, in turn, passes back to back:
// prefill 32 x 16384 x 64 546 -> 529 us, step of 16 heads x 12287 855 -> 838, forward of 32 x 4096 62.5 -> 60.1, smooth step 32 x 16384 629 -> 624.
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);      // (its error is the one that HA_LAUNCHED finds)
}
// Lets the CTAs of a chained kernel that comes next be placed as soon as all of this kernel's are.
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// First statement of every thread of a chained kernel: waits until the previous kernel is complete and its memory operations are visible.  Nothing is
// read or written before it, so that what lies further back in the stream is complete, too.
__device__ __forceinline__ void chain_begin() {
  chain_release();
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

inline int dtype_size(int dtype) { return dtype == HA_FP32 ? 4 : 2; }

// n / d for 0 <= n < 2^31 by one wide multiplication and a shift (m = ceil(2^(31 + s) / d), s = ceil(log2 d): the round-up method).
struct FastDiv {
  uint32_t m = 1u << 31, s = 0;
  FastDiv() = default;
  explicit FastDiv(uint32_t d) {
    while ((1ull << s) < d) ++s;
    m = (uint32_t)(((1ull << (31 + s)) + d - 1) / d);
  }
  __host__ __device__ __forceinline__ int operator()(int n) const { return (int)(((unsigned long long)(uint32_t)n * m) >> (31 + s)); }
};

// Number of SMs of the current device, looked up once per device.
inline int sm_count() {
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 148;
  int v = cache[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    cache[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

// Opt-in dynamic shared memory size of a kernel: a per-device function attribute, set at the first launch on each device
// (one process may drive several GPUs) instead of before every launch.
#define HA_SMEM_ATTR_ONCE(kernel, bytes, where)                                                        \
  do {                                                                                                 \
    static std::atomic<unsigned long long> _done{0};                                                   \
    int _dev = 0;                                                                                      \
    cudaGetDevice(&_dev);                                                                              \
    const unsigned long long _bit = 1ull << (_dev & 63);                                               \
    if (!(_done.load(std::memory_order_acquire) & _bit)) {                                             \
      HA_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), where); \
      _done.fetch_or(_bit, std::memory_order_release);                                                 \
    }                                                                                                  \
  } while (0)

// Dynamic shared memory of a kernel whose layout of `used` bytes starts at the first 1 KB boundary after its static variables: looked up at the
// first launch (by whichever host thread comes first; they all find the same).
#define HA_WINDOW_BYTES(bytes, kernel, used, where)                                                    \
  do {                                                                                                 \
    static std::atomic<int> _bytes{0};                                                                 \
    bytes = _bytes.load(std::memory_order_relaxed);                                                    \
    if (bytes == 0) {                                                                                  \
      cudaFuncAttributes _fa;                                                                          \
      HA_CUDA_OK(cudaFuncGetAttributes(&_fa, kernel), where);                                          \
      const int _stat = ((int)_fa.sharedSizeBytes + 15) / 16 * 16;                                     \
      bytes = (1024 - _stat % 1024) % 1024 + (used);                                                   \
      _bytes.store(bytes, std::memory_order_relaxed);                                                  \
    }                                                                                                  \
  } while (0)

// ---------------------------------------------------------------------------------------------------
// element access
// ---------------------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// value of v after a round trip through T (used where the reference rounds an intermediate to the input dtype)
template <typename T> __device__ __forceinline__ float round_to(float v) { return to_f32<T>(from_f32<T>(v)); }

template <typename T> __device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <typename T> __device__ __forceinline__ float2 unpack2(uint32_t w);
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
template <> __device__ __forceinline__ float2 unpack2<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<__half2*>(&w));
}

// ---------------------------------------------------------------------------------------------------
// PTX wrappers: shared addresses, mbarrier, cp.async, tcgen05
// ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
// Bounded wait: returns false when the phase did not complete within SPIN_LIMIT polls or WAIT_CYCLES cycles.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (int i = 0; i < SPIN_LIMIT; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > WAIT_CYCLES) return false;
  }
  return false;
}

// The same inside a kernel whose roles share an abort flag: whoever gives up raises it, everybody else leaves at the next wait.
// (A poll may itself suspend the thread for a while; the time cap, about a second, is what bounds the wait.)
__device__ __forceinline__ bool mbar_wait_or_abort(uint32_t bar, uint32_t parity, int* abort_flag) {
  if (__builtin_expect(mbar_try_wait(bar, parity), 1)) return true;
  const uint32_t t0 = (uint32_t)clock();
#pragma unroll 1
  while (!mbar_try_wait(bar, parity)) {
    if ((uint32_t)clock() - t0 > (uint32_t)WAIT_CYCLES) *reinterpret_cast<volatile int*>(abort_flag) = 1;
    if (*reinterpret_cast<volatile int*>(abort_flag)) return false;
  }
  return true;
}

// 16-byte async copy global -> shared; src_bytes = 0 zero-fills the destination.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// makes generic-proxy writes to shared memory visible to the async proxy (tcgen05.mma operand reads)
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t slot_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle, version 1 (sm_100).  Operand tiles are stored as slabs of
// rows x 128 bytes, each 8-row group occupying 1024 contiguous bytes with 16-byte chunk c of row r at chunk
// position c ^ (r & 7).
//  * K-major use (rows = M or N index, 64 elements of K per slab): lbo unused, sbo = 1024, one K=16 step
//    advances the start address by 32 bytes, the next slab holds the next 64 K-elements.
//  * MN-major use (rows = K index, 64 elements of M/N per slab): sbo = 1024 (next 8 K-rows), lbo = slab stride
//    (next 64 M/N elements), one K=16 step advances the start address by 2048 bytes.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// byte offset of element (row, col) inside a swizzled slab tile; col in elements of 2 bytes, slab_rows rows per slab
__device__ __forceinline__ uint32_t swz_off(int slab_rows, int row, int col) {
  return (uint32_t)((col >> 6) * (slab_rows * 128) + row * 128 + ((((col >> 3) & 7) ^ (row & 7)) << 4) + (col & 7) * 2);
}

// Instruction descriptor for kind::f16: fp32 accumulate, A/B both bf16 (ab_fmt = 1) or fp16 (0).
__device__ __forceinline__ uint32_t mma_idesc(int M, int N, int ab_fmt, int a_mn_major, int b_mn_major) {
  return (1u << 4) | ((uint32_t)ab_fmt << 7) | ((uint32_t)ab_fmt << 10) | ((uint32_t)a_mn_major << 15) |
         ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One lane of the (converged) warp, always the same one.  Around tcgen05 instructions in warp-uniform code it lets the compiler keep
// descriptors in uniform registers; a `lane == 0` branch does not (measured: 64 against 126 cycles per N = 128 instruction).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred P;\n .reg .b32 R;\n elect.sync R|P, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, P;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// For a CTA that gave up: waits (bounded) for the products that this warp's elected lane has issued.  `bar`: one arrival, used for nothing else.
__device__ __forceinline__ void mma_settle(uint32_t bar) {
  __syncwarp();
  if (elect_one()) mma_commit(bar);
  __syncwarp();
  mbar_wait(bar, 0);
}

// 32 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_fence16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
// 16 TMEM lanes x 32 columns as four fragments of 16 x 8: registers 4 j + 2 k, + 1 hold columns 8 j + 2 (lane % 4), + 1 of TMEM lane 8 k + lane / 4
__device__ __forceinline__ void tmem_ld_16x256(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// ... 16 TMEM lanes x 16 columns: register 2 j + k to column 4 j + lane % 4 of TMEM lane 8 k + lane / 4
__device__ __forceinline__ void tmem_st_16x128(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// four 8 x 8 matrices of 16-bit elements: lane l names row l % 8 of matrix l / 8 (16 bytes), register m holds its elements of matrix m
__device__ __forceinline__ void store_matrix_x4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// Waits for this thread's outstanding tcgen05.ld; the loaded registers are passed through the statement so that
// no use of them can be scheduled ahead of the wait.
__device__ __forceinline__ void tmem_ld_fence(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                 "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                 "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// Packed pairs of fp32 (sm_100 executes fma/add/mul on two floats per instruction)
__device__ __forceinline__ uint64_t pack_f2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack_u2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}


// Optional per-phase cycle counters of the attention kernels (compiled in only with -DHA_PHASE_TIMING; the counters
// of the first CTAs are written to the buffer registered with ha_debug_set_timing_buffer_fwd / _bwd).
#ifdef HA_PHASE_TIMING
static __device__ unsigned long long* g_timing_buf = nullptr;   // one per translation unit
#define HA_T_SETTER(name) extern "C" int name(void* buf) { return cudaMemcpyToSymbol(::ha::g_timing_buf, &buf, sizeof(buf)) == cudaSuccess ? 0 : -4; }
#define HA_T_DECL(n) long long _t_acc[n] = {0}; long long _t_last = clock64();
#define HA_T_MARK(i) { long long _t_now = clock64(); _t_acc[i] += _t_now - _t_last; _t_last = _t_now; }
#define HA_T_DUMP(n, cta, cond) if ((cond) && g_timing_buf && (cta) < 4096) { for (int _i = 0; _i < n; ++_i) g_timing_buf[(cta) * 16 + _i] = _t_acc[_i]; }
#else
#define HA_T_SETTER(name)
#define HA_T_DECL(n)
#define HA_T_MARK(i)
#define HA_T_DUMP(n, cta, cond)
#endif

// A bounded wait gave up: record it in the device status word and, if the caller gave one, in the host-visible word.
__device__ __forceinline__ void report_status(int32_t* status, int32_t* status_host, int32_t code) {
  if (status) atomicExch(status, code);
  if (status_host) {
    *reinterpret_cast<volatile int32_t*>(status_host) = code;
    __threadfence_system();
  }
}
__device__ __forceinline__ void report_timeout(int32_t* status, int32_t* status_host) { report_status(status, status_host, HA_DEV_TIMEOUT); }
// Did an earlier CTA of this (or a previous) launch give up?  One thread reads the word and the whole CTA branches on
// the shared copy, so the answer is the same for every thread even while another CTA is writing the word.
// Contains a __syncthreads(): call it from every thread of the CTA.
__device__ __forceinline__ bool cta_sees_failure(const int32_t* status, int* s_flag) {
  if (threadIdx.x == 0) *s_flag = status ? *reinterpret_cast<const volatile int32_t*>(status) : 0;
  __syncthreads();
  return *s_flag != 0;
}

// pulls the 128-byte line holding `p` into L2 without blocking the thread
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^x of two values on the FMA and integer pipes, for the share of a softmax's exponentials that the exponential unit (four lanes a clock
// and scheduler) cannot take: x = n + f with n the nearest integer (Cody-Waite, by adding and subtracting 1.5 * 2^23 + 127, which
// leaves n + 127, the exponent field of 2^n, in the low bits), 2^f on [-1/2, 1/2] by a degree 5 polynomial with value 1 at 0 whose
// largest relative error is minimal (found as a linear programme over 4001 Chebyshev points; 1.7e-7 in fp32 arithmetic, the exponential
// unit's own bound is 2.4e-7), the two multiplied.  Arguments up to 127; below -127, -infinity among them, they give 0.  A NaN stays
// one: the clamp hands it on and the product keeps it, whatever its exponent field became.
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void poly_exp2_2(uint64_t x2, float& lo, float& hi) {
  float a, b;
  unpack_f2(x2, a, b);
  x2 = pack_f2(max_nan(a, -127.f), max_nan(b, -127.f));
  const uint64_t magic = pack_f2(12583039.f, 12583039.f), nmagic = pack_f2(-12583039.f, -12583039.f), mone = pack_f2(-1.f, -1.f);
  const uint64_t r = fadd2(x2, magic);
  const uint64_t f = ffma2(fadd2(r, nmagic), mone, x2);
  auto c = [](float v) { return pack_f2(v, v); };
  uint64_t q = ffma2(f, c(0x1.5bba14p-10f), c(0x1.3cea88p-7f));
  q = ffma2(f, q, c(0x1.c6b752p-5f));
  q = ffma2(f, q, c(0x1.ebf9bcp-3f));
  q = ffma2(f, q, c(0x1.62e42ap-1f));
  q = ffma2(f, q, c(1.f));
  unpack_f2(r, a, b);
  unpack_f2(fmul2(q, pack_u2(__float_as_uint(a) << 23, __float_as_uint(b) << 23)), lo, hi);
}

}  // namespace ha
