// Internal declarations shared by the CUDA translation units of libb3gpu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <vector>

#include "../../include/b3gpu.h"

// ---------------------------------------------------------------------------
// Error reporting
// ---------------------------------------------------------------------------
void b3_set_error(const char* fmt, ...);

#define B3_CUDA(call)                                                          \
    do {                                                                       \
        cudaError_t e__ = (call);                                              \
        if (e__ != cudaSuccess) {                                              \
            b3_set_error("%s:%d %s -> %s", __FILE__, __LINE__, #call,          \
                         cudaGetErrorString(e__));                             \
            return B3_ERR_CUDA;                                                \
        }                                                                      \
    } while (0)

#define B3_CHECK_LAUNCH()                                                      \
    do {                                                                       \
        cudaError_t e__ = cudaGetLastError();                                  \
        if (e__ != cudaSuccess) {                                              \
            b3_set_error("%s:%d launch -> %s", __FILE__, __LINE__,             \
                         cudaGetErrorString(e__));                             \
            return B3_ERR_CUDA;                                                \
        }                                                                      \
    } while (0)

#define B3_TRY(expr)                                                           \
    do {                                                                       \
        int s__ = (expr);                                                      \
        if (s__ != B3_OK) return s__;                                          \
    } while (0)

struct b3Context_t {
    int device = 0;
    int numSMs = 148;
    int maxSmemOptin = 0;
    // scratch for the primitive entry points (grown on demand)
    void* scratch = nullptr;
    size_t scratchBytes = 0;
    int ensureScratch(size_t bytes);
};

static inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Lets a kernel take all the dynamic shared memory that a block can have. The
// attribute is the function's, on its device, and not a world's: every caller sets
// the same value, so that none lowers it between another thread's set and launch.
static inline int allow_dynamic_smem(b3Context ctx, const void* kern) {
    cudaFuncAttributes a;
    B3_CUDA(cudaFuncGetAttributes(&a, kern));
    B3_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 ctx->maxSmemOptin - (int)a.sharedSizeBytes));
    return B3_OK;
}

// ---------------------------------------------------------------------------
// Device-wide primitives (implemented in primitives.cu). All take a device
// side element count (n_dev) so they can be captured in CUDA graphs without
// host synchronisation; n_max bounds the grid and scratch sizes, and is the
// count itself where n_dev is null. n_expect (0: n_max) is the likely count.
// cleared: the scratch is cleared already (a sort's first 16 bytes, by a kernel
// after the last sort; all of a scan's, with other buffers).
// ---------------------------------------------------------------------------
namespace b3 {

// Polls of a device-side wait before it gives up (the Jacobi grid barrier's
// limit can be changed per world, b3_set_wait_limits).
constexpr int kDefaultSpinLimit = 1 << 22;

// Radix sort scratch: bytes for n_max elements.
size_t radix_scratch_bytes(int64_t n_max, int key_bits);
// Sort (keys, vals) of device count *n_dev (<= n_max). The sorted result
// ends in (keys_alt, vals_alt) or in (keys, vals); *result_in_alt tells which. vals may be null (keys only).
bool radix_result_in_alt(int64_t n_max, int key_bits);  // what *result_in_alt will be
int radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt,
                     const int32_t* n_dev, int64_t n_max, int key_bits, void* scratch,
                     size_t scratch_bytes, int32_t* err_flag, cudaStream_t st, bool* result_in_alt,
                     int numSMs, int64_t n_expect = 0, bool cleared = false);

// Out-of-place sort: (keys_in, vals_in) are only read; the sorted result
// lands in (keys_out, vals_out); (keys_tmp, vals_tmp) hold the passes in
// between (unused for one pass). vals_in may be null (keys only).
int radix_sort_kv_out(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                      uint32_t* keys_tmp, uint32_t* vals_tmp, const int32_t* n_dev, int64_t n_max, int key_bits,
                      void* scratch, size_t scratch_bytes, int32_t* err_flag, cudaStream_t st, int numSMs,
                      bool cleared = false);
// Interleaved (key, value) pairs (btSortData): result in kv_alt when
// *result_in_alt, else in kv.
int radix_sort_interleaved(uint2* kv, uint2* kv_alt, const int32_t* n_dev, int64_t n_max, int key_bits,
                           void* scratch, size_t scratch_bytes, int32_t* err_flag, cudaStream_t st,
                           bool* result_in_alt, int numSMs, bool cleared = false);

size_t scan_scratch_bytes(int64_t n_max);
// Exclusive scan of n_dev u32 values; total to d_total (may be null).
int exclusive_scan_u32(const uint32_t* src, uint32_t* dst, const int32_t* n_dev, int64_t n_max,
                       uint32_t* d_total, void* scratch, size_t scratch_bytes, int32_t* err_flag,
                       cudaStream_t st, int numSMs, bool cleared = false);

int fill_u32(uint32_t* dst, uint32_t v, int64_t n, cudaStream_t st);
int bound_search(const uint32_t* keys, const int32_t* n_dev, int64_t n_max, uint32_t* dst,
                 int64_t n_dst, int mode, cudaStream_t st);
int bound_search_interleaved(const uint2* kv, const int32_t* n_dev, int64_t n_max, uint32_t* dst, int64_t n_dst,
                             int mode, cudaStream_t st);

}  // namespace b3

// ---------------------------------------------------------------------------
// Device helpers
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
namespace b3dev {

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Bounded spin budget for every device-side wait: about 4M polls with a
// short back-off (well under a second), after which the waiter records an
// error and proceeds instead of hanging the GPU.
constexpr int kSpinLimit = b3::kDefaultSpinLimit;

// Grid barrier of a cooperative launch. Blocks add to one 64-bit word with a
// release and poll it with an acquire until all of this round have arrived;
// the count only grows within a launch (the host clears it before), so no
// second word has to be released and a wait ends one L2 round trip after the
// last arrival. A waiter gives up after spinLimit polls: it sets *err, counts
// a timeout and sets the word's top bit, on which every block leaves at this
// or its next barrier, so the launch always ends. heed: an error that was set
// before the launch ends it at the first barrier too (the solves, whose results
// are void by then). A sort pays no heed to it: it is the host that clears an
// error, steps go on until then, and what they index with is a sort's output.
struct GridBarrier {
    unsigned long long* word;
    unsigned long long target;
    int32_t* err;
    b3Counters* counters;
    int spinLimit;
    int before;  // thread 0: *err at the kernel's start, where that is heeded
    unsigned blocks;  // that take part, block 0 on

    __device__ __forceinline__ GridBarrier(uint32_t* w, int32_t* e, b3Counters* c, int limit, bool heed,
                                           unsigned taking = gridDim.x)
        : word(reinterpret_cast<unsigned long long*>(w)), target(0), err(e), counters(c), spinLimit(limit), before(0),
          blocks(taking) {
        if (heed && threadIdx.x == 0) before = *(volatile int32_t*)e;
    }
    __device__ __forceinline__ bool wait() {
        constexpr unsigned long long kAbort = 1ull << 63;
        int ok = 1;
        target += blocks;
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(word), "l"(1ull) : "memory");
            unsigned long long v = ld_acquire_u64(word);
            for (int spins = 0; !(v & kAbort) && v < target; v = ld_acquire_u64(word)) {
                if (++spins > spinLimit) {
                    atomicExch(err, 1);
                    if (counters) atomicAdd(&counters->timeouts, 1);
                    atomicOr(word, kAbort);
                    v = kAbort;
                    break;
                }
                if (spins > 16) __nanosleep(64);
            }
            ok = !(v & kAbort) && before == 0;
        }
        return __syncthreads_and(ok) != 0;
    }
};

// 16 bytes read or written as one: a reader sees a record whole, of one version
// or another, so a version number in it says that the rest is of that version.
__device__ __forceinline__ float4 ld_whole(const float4* p) {
    unsigned long long lo, hi;
    asm volatile(
        "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
        : "=l"(lo), "=l"(hi)
        : "l"(p)
        : "memory");
    return make_float4(__uint_as_float((uint32_t)lo), __uint_as_float((uint32_t)(lo >> 32)),
                       __uint_as_float((uint32_t)hi), __uint_as_float((uint32_t)(hi >> 32)));
}
__device__ __forceinline__ void st_whole(float4* p, float4 v) {
    const unsigned long long lo = __float_as_uint(v.x) | (unsigned long long)__float_as_uint(v.y) << 32;
    const unsigned long long hi = __float_as_uint(v.z) | (unsigned long long)__float_as_uint(v.w) << 32;
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(lo), "l"(hi)
                 : "memory");
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

}  // namespace b3dev
#endif
