// Shared declarations of the library: device object, error reporting, dtype helpers.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <vector>

#include "../../include/autograph_b200.h"

namespace ag {

// ---- error reporting -----------------------------------------------------
// Thread-local message behind ag_last_error().
char *error_buffer();
int fail(int status, const char *fmt, ...) __attribute__((format(printf, 2, 3)));

#define AG_CUDA_TRY(expr)                                                                      \
    do {                                                                                       \
        cudaError_t _e = (expr);                                                               \
        if (_e != cudaSuccess) {                                                               \
            /* reported here: it must not also fail the next call's launch check */           \
            cudaGetLastError();                                                                \
            return ::ag::fail(_e == cudaErrorMemoryAllocation ? AG_ERR_OOM : AG_ERR_CUDA,      \
                              "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, \
                              __LINE__);                                                       \
        }                                                                                      \
    } while (0)

#define AG_TRY(expr)              \
    do {                          \
        int _s = (expr);          \
        if (_s != AG_OK) return _s; \
    } while (0)

#define AG_REQUIRE(cond, status, ...)                   \
    do {                                                \
        if (!(cond)) return ::ag::fail(status, __VA_ARGS__); \
    } while (0)

// Counts kernel launches enqueued by the library (ag_kernel_launch_count).
void count_launch();
void count_launches(uint64_t n);
uint64_t launch_count();

// Checks the launch that was just enqueued.
#define AG_CHECK_LAUNCH()                  \
    do {                                   \
        ::ag::count_launch();              \
        AG_CUDA_TRY(cudaGetLastError());   \
    } while (0)

}  // namespace ag

// Tiles whose k slices may be added by the CTA that finishes last.
constexpr int kTileCounters = 1024;

// ---- device object ---------------------------------------------------------
// One per (GPU, stream).  Owns a scratch workspace that kernels such as the
// split-k GEMM use for partial sums, a device status word that bounded device
// waits report into, and a pinned host word for scalar read-backs.
struct ag_device {
    int ordinal = 0;
    cudaStream_t stream = nullptr;
    bool owns_stream = false;
    int sm_count = 0;
    std::recursive_mutex mu;
    void *workspace = nullptr;
    size_t workspace_bytes = 0;
    void *staging = nullptr;        // second scratch block: operand re-layouts of the
    size_t staging_bytes = 0;       // tensor-core convolution (may be live next to workspace)
    void *engine = nullptr;         // third block: k-slice sums and packed operands of the
    size_t engine_bytes = 0;        // tensor-core engines (live next to the other two)
    std::vector<void *> retired;    // outgrown scratch blocks that captured graphs may still use
    int *tile_counters = nullptr;   // kTileCounters zeros: arrivals at a tile, back to zero after each launch
    int *status_dev = nullptr;      // device word: 0 = ok, else a timeout code
    int *status_host = nullptr;     // pinned mirror
    float *scalar_dev = nullptr;    // small device buffer for loss / accuracy sums (64 B)
    float *scalar_host = nullptr;   // pinned mirror
    // Completion of a blocking call's last kernel, written by the kernel itself (see signal_done).
    volatile uint32_t *done_host = nullptr;
    uint32_t *done_dev = nullptr;   // the same word as the device sees it
    uint32_t done_seq = 0;
    uint32_t signal = 0;            // not 0: the next kernel that can signal takes it and clears it
};

namespace ag {

// Programmatic dependent launch.  A kernel launched with launch_dependent may be placed on SMs that its
// predecessor in the stream has left and set itself up there; after dependency_wait everything the
// predecessor wrote is visible.  Every thread that touches global memory comes through that wait first.
// That holds for loads through the read-only path too (__ldg, const __restrict__), which most operators use: they
// rely on no line of what the predecessor writes coming into an SM's L1 between its write and their wait, and
// nothing loads such data earlier.
// A kernel that allocates tensor memory does so before it lets dependents launch: one that came first could hold the
// columns it still needs, and wait for it.
// The operators' kernels are small enough for that to count: a kernel of 2 us in a stream of them took 4 us, and a
// convolution stage called operator by operator (16 -> 32 3x3, 64 x 32 x 32 f32, eleven launches) 118 us, now 100.
//
// Grids of up to half of the SMs let their dependents launch at once: those find the other half free.  Larger ones
// say nothing, and their dependents launch when the last of their CTAs ends.  Let go at their start, dependents, and
// theirs, took what room there was on the SMs that came free first and left the others idle, most of all replayed
// from a graph, where no launch holds them up (us at the start, at the end): f32 256^3 13.0, 8.3; bf16 16 x 64 x 31 x 31
// -> 128 3x3 24.2, 14.9; training LeNet5's layers on 2000 images bf16 518, 348.  Up to 111 CTAs at the start is too many
// (convolution 1 -> 6 5x5, 100 x 28 x 28 f32: 4.7, 3.6); none at all costs small chains (LeNet5's layers, 16 images: 24.8
// for 22.8 us an inference).
// kAlwaysEarly: kernels that are followed by ones of a CTA per SM, which cannot crowd and gain their set-up time -- the
// layout, filter and gradient passes around the tensor-core convolutions, the gathered engine's products (a training step
// of the wide stack, 256 images bf16: 491 us without, 482 with; 65536 x 512 x 16 f32 103.5 and 101.0).
constexpr unsigned kEarlyCtas = 74, kAlwaysEarly = ~0u;
__device__ __forceinline__ void let_dependents_launch(unsigned most = kEarlyCtas) {
    if (gridDim.x * gridDim.y * gridDim.z <= most) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
int launch_dependent(ag_device *dev, void (*kernel)(P...), dim3 grid, dim3 threads, size_t smem, const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = dev->stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    AG_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
    AG_CHECK_LAUNCH();
    return AG_OK;
}

// How a kernel tells a waiting host thread that it is done: its last CTA writes `seq` to a word of pinned
// memory, which the host polls.  cudaStreamSynchronize returns 3 us later (launch and wait 10.5 us, with
// the word 7.4), a sixth of a small inference call.
struct Done {
    uint32_t *flag = nullptr;       // null: nobody waits
    int *arrivals = nullptr;        // a zero, back to zero afterwards
    uint32_t seq = 0;
};
inline Done take_signal(ag_device *dev) {
    Done d;
    if (dev->signal != 0) {
        d.flag = dev->done_dev;
        d.arrivals = dev->tile_counters + kTileCounters - 1;
        d.seq = dev->signal;
        dev->signal = 0;
    }
    return d;
}
// Arms the next kernel that can signal; false when there is nothing to poll.
inline bool arm_signal(ag_device *dev) {
    if (dev->done_host == nullptr) return false;
    if (++dev->done_seq == 0) ++dev->done_seq;
    dev->signal = dev->done_seq;
    return true;
}
// Waits for the work of an armed call: by the word if a kernel took the signal, else (or when the word
// does not come within 20 ms, as after an error) by the stream.
cudaError_t wait_signal(ag_device *dev, bool armed);

// Called by all threads of every CTA, after their last stores.
__device__ __forceinline__ void signal_done(const Done &d) {
    if (d.flag == nullptr) return;
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence_system();
    if (gridDim.x > 1) {
        if (atomicAdd(d.arrivals, 1) != (int)gridDim.x - 1) return;
        *d.arrivals = 0;
        __threadfence_system();
    }
    *reinterpret_cast<volatile uint32_t *>(d.flag) = d.seq;
}

// Makes `dev` current on the calling thread and locks it for the call.
class DeviceGuard {
   public:
    explicit DeviceGuard(ag_device *dev) : lock_(dev->mu) { err_ = cudaSetDevice(dev->ordinal); }
    cudaError_t error() const { return err_; }

   private:
    std::lock_guard<std::recursive_mutex> lock_;
    cudaError_t err_;
};

#define AG_ENTER(dev)                                                                     \
    AG_REQUIRE((dev) != nullptr, AG_ERR_INVALID, "device is null");                       \
    ::ag::DeviceGuard _guard(dev);                                                        \
    if (_guard.error() != cudaSuccess)                                                    \
    return ::ag::fail(AG_ERR_CUDA, "cudaSetDevice(%d) failed: %s", (dev)->ordinal,        \
                      cudaGetErrorString(_guard.error()))

// Returns a workspace of at least `bytes` (grown on demand; outgrown blocks stay allocated
// until the device is destroyed because captured graphs may still point into them).
int workspace(ag_device *dev, size_t bytes, void **out);
// The same for the second scratch block.
int staging(ag_device *dev, size_t bytes, void **out);
// The same for the tensor-core engines' block: a product may run on operands that lie in either of
// the other two.
int engine_scratch(ag_device *dev, size_t bytes, void **out);

inline size_t dtype_size(ag_dtype t) {
    switch (t) {
        case AG_F32: return 4;
        case AG_BF16: return 2;
        case AG_U8: return 1;
        case AG_U16: return 2;
        case AG_U32: return 4;
    }
    return 0;
}

inline bool is_float_dtype(ag_dtype t) { return t == AG_F32 || t == AG_BF16; }
inline bool is_label_dtype(ag_dtype t) { return t == AG_U8 || t == AG_U16 || t == AG_U32; }

// ---- element conversion (device) ------------------------------------------
__device__ __forceinline__ float to_f32(float x) { return x; }
// A shift of the bits.
__device__ __forceinline__ float to_f32(__nv_bfloat16 x) { return __uint_as_float((uint32_t)__bfloat16_as_ushort(x) << 16); }
// An operand's element, or zero outside of it: a load under a predicate, so that several can be in flight
// (256 x 200 x 10, transposed: f32 11.5 us with a branch around each, 10.7 so; bf16 26.2 and 23.9).
__device__ __forceinline__ float load_or_zero(const float *p, bool ok) {
    float v = 0.f;
    if (ok) v = __ldg(p);
    return v;
}
__device__ __forceinline__ float load_or_zero(const __nv_bfloat16 *p, bool ok) {
    uint32_t v = 0;
    if (ok) v = __ldg(reinterpret_cast<const unsigned short *>(p));
    return __uint_as_float(v << 16);
}
template <class T>
__device__ __forceinline__ T from_f32(float x);
template <>
__device__ __forceinline__ float from_f32<float>(float x) {
    return x;
}
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) {
    return __float2bfloat16_rn(x);
}

// Unsigned division by a runtime constant without a divide instruction.
// Valid for dividends below 2^31.
struct FastDiv {
    uint32_t d = 1, mul = 0, shr = 0;
    FastDiv() = default;
    explicit FastDiv(uint32_t divisor) : d(divisor) {
        if (divisor <= 1) {
            d = 1;
            return;
        }
        uint32_t l = 0;
        while ((1ull << l) < divisor) ++l;  // ceil(log2 d)
        uint64_t p = 31 + l;
        mul = (uint32_t)(((1ull << p) + divisor - 1) / divisor);
        shr = l - 1;
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const {
        return d == 1 ? n : (__umulhi(n, mul) >> shr);
    }
    __device__ __forceinline__ void divmod(uint32_t n, uint32_t &q, uint32_t &r) const {
        q = div(n);
        r = n - q * d;
    }
};

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Dynamic shared memory of a persistent kernel that wants an SM per CTA.  Launched while its predecessor still runs, its
// CTAs go to the SMs that came free first, two or three to one if they fit, and the others stay idle (after kernels that
// let dependents launch at their start, the wide stack at 256 images bf16: inference 203 us, so 289, a training step 492
// and 569): more than half of an SM's memory keeps them apart.
constexpr int kOneCtaPerSm = 116 * 1024;

// What lets a kernel have more than 48 KB of dynamic shared memory is an attribute of the (kernel, GPU) pair, while calls are
// serialised per ag_device: devices of one GPU in several threads share it.  So every kernel gets one constant that no
// call exceeds.  A size per call, or the largest so far, can be lowered by another thread between a call's set and its
// launch, which then fails.
constexpr int kMostSmem = 226 * 1024;   // of 227, beside up to 1 KB of static shared memory
struct SmemAllowed {
    std::atomic<uint64_t> gpus{0};   // a bit per ordinal; beyond 64 of them the attribute is set on every call
};
template <int MOST = kMostSmem, class K>
int allow_smem(ag_device *dev, K kernel, SmemAllowed &done) {
    const uint64_t bit = dev->ordinal < 64 ? 1ull << dev->ordinal : 0;
    if (done.gpus.load(std::memory_order_acquire) & bit) return AG_OK;
    AG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST));
    done.gpus.fetch_or(bit, std::memory_order_release);
    return AG_OK;
}

}  // namespace ag
