// Shared helpers of the sm_100a kernels: error reporting through a C ABI, dtype codes,
// loads that widen to float, warp/block reductions with a fixed order.
//
// Every exported function is `extern "C" int ember_<name>(..., void* stream)`: it
// validates its arguments on the host, launches on the given stream, and returns 0 or a
// non-zero code with a message readable through ember_last_error().  Kernels never trap:
// an index that is out of range is skipped and recorded in a device error word that the
// host can poll.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <utility>

#define EMBER_API extern "C" __attribute__((visibility("default")))

enum EmberDType : int { EMBER_F32 = 0, EMBER_BF16 = 1 };

// Device error word bits (set with atomicOr by kernels, read by the host after a sync).
enum EmberDeviceError : int {
    EMBER_ERR_TOKEN_RANGE = 1,   // a token id outside the vocabulary
    EMBER_ERR_PAGE_RANGE = 2,    // a page id outside the pool
    EMBER_ERR_WAIT_LIMIT = 4,    // a bounded wait on a barrier ran out
};

namespace ember {

inline char* error_buffer() {
    static thread_local char buf[512] = {0};
    return buf;
}

inline int fail(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(error_buffer(), 512, fmt, ap);
    va_end(ap);
    return 1;
}

inline int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail("%s: %s", what, cudaGetErrorString(e));
    return 0;
}

// Programmatic dependent launch.  Every kernel is launched with the stream-serialization attribute,
// so its blocks may start while the kernel before it is still draining; until pdl_wait() returns a
// kernel touches nothing that an earlier kernel of the step writes.  It may set up barriers, read the step's uploaded
// integers and prefetch what its caller says is settled: weights, and the keys of earlier steps.  The one exception acquires a
// ticket instead (below).
// pdl_wait() returns at once when the launch carried no such dependency.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A kernel that is to run beside the one in front of it (attention_tc.cu beside attention_fa.cu) cannot wait for that one,
// and launch_dependents orders no memory.  So the one in front, behind its own pdl_wait(), stores a ticket with release
// semantics, and the other reads it with acquire semantics: all that the first had waited for happens before what the second
// does then (other threads of its block: behind a block barrier).  Each launch has a ticket of its own, and who does not
// find it waits with pdl_wait(): this decides, it never spins.
__device__ __forceinline__ void release_ticket(int* at, int ticket) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(at), "r"(ticket) : "memory");
}
__device__ __forceinline__ int acquire_ticket(const int* at) {
    int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(at) : "memory");
    return v;
}
// A captured launch that looks for a ticket would find the one of the replay before: it is given none.
inline bool is_capturing(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) { cudaGetLastError(); return true; }
    return status != cudaStreamCaptureStatusNone;
}

inline bool pdl_enabled() {
    static int on = -1;
    if (on < 0) {
        const char* e = getenv("EMBER_PDL");
        on = (e && e[0] == '0') ? 0 : 1;
    }
    return on != 0;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                 Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// ---- bounded waits on shared-memory barriers ------------------------------------------------------------------
// No kernel here waits without a limit.  A wait gives up after EMBER_WAIT_LIMIT_NS of the device's global timer
// (two seconds: far beyond any step, short enough that nobody takes the device for hung), raises the block's
// abort flag so that every role of the block falls through to the common exit (which frees tensor memory and
// records EMBER_ERR_WAIT_LIMIT in the device error word), and returns false.  The limit is time, not a number of
// polls: a suspended try_wait takes an implementation-defined while, so a poll count bounds nothing in seconds.
constexpr unsigned long long EMBER_WAIT_LIMIT_NS = 2000000000ull;

__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbarrier_try_wait_parity(uint32_t bar_shared, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(bar_shared), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbarrier_test_wait_parity(uint32_t bar_shared, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(bar_shared), "r"(parity) : "memory");
    return ok != 0;
}
// A phase that is already over is seen by one plain look (about 100 cycles; the suspending form costs about 240
// even then).  While waiting, the abort flag and the timer are looked at every 64 polls.
__device__ __forceinline__ bool mbarrier_wait_bounded(uint32_t bar_shared, uint32_t parity, volatile int* abort_flag,
                                                      unsigned long long limit_ns = EMBER_WAIT_LIMIT_NS) {
    if (mbarrier_test_wait_parity(bar_shared, parity)) return true;
    unsigned long long start = 0;
    for (unsigned i = 0;; i++) {
        if (mbarrier_try_wait_parity(bar_shared, parity)) return true;
        if ((i & 63u) == 63u) {
            if (*abort_flag) return false;
            const unsigned long long now = global_timer_ns();
            if (start == 0) start = now;
            else if (now - start > limit_ns) break;
        }
    }
    *abort_flag = 1;
    return false;
}

// One lane of a warp whose lanes are all here, the same one each time.  What issues tensor instructions and TMA copies goes
// through its loops as a whole warp and elects the lane that issues: the control flow then is uniform, and so are the registers
// that these instructions take their operands from.  A lane singled out by its number pays for moving each operand there
// (attention: 77 cycles an MMA of 128 x 64 x 16 against 56; products, us before -> now: 2,048 tokens x 12,288 x 2,048 gated
// 79.4 -> 71.4, x 24,576 x 4,096 gated 293 -> 265, 601 tokens x 4,096 x 2,048 14.7 -> 13.2, 8 tokens x 2,048 x 6,144 7.2 -> 6.9;
// a look at the next stage's barrier ahead of the issue gains nothing more).
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(one));
    return one != 0;
}
// The warp's number, known to be the same in all its lanes.
__device__ __forceinline__ int warp_number() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ float to_float(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T>
__device__ __forceinline__ T from_float(float x);
template <>
__device__ __forceinline__ float from_float<float>(float x) { return x; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

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

// Sum over a block of up to 1024 threads; the order of additions is fixed by the
// thread layout, so the result does not depend on anything but the inputs.
__device__ __forceinline__ float block_sum(float v, float* scratch /* >= 32 floats */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    const int nwarps = (blockDim.x + 31) >> 5;
    float r = (lane < nwarps) ? scratch[lane] : 0.0f;
    r = warp_sum(r);
    return r;
}

}  // namespace ember

// Each shared library exports its own copy of the message reader.
#define EMBER_DEFINE_LAST_ERROR \
    EMBER_API const char* ember_last_error() { return ember::error_buffer(); }
