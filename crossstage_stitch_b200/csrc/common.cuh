// Shared host/device helpers for the stage kernels (sm_100a).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <climits>
#include <cstddef>
#include <cstdint>

#include "stage_api.hpp"

namespace stitch::b200 {

constexpr std::size_t kWorkspaceAlign = 256;
constexpr int kSmCount = 148;  // B200: grid sizing target, not a correctness input

// Kernel launches issued by this library (all threads, all devices); read
// through stitch_launch_count() to attribute device work to these kernels.
void note_launches(int n);

// Launches of the per-image and per-pair calls: a kernel may be scheduled while
// the one before it on the stream still runs, and holds at
// wait_for_previous() until that one has completed and its writes are visible.
// Before the wait a kernel reads its launch parameters and constant tables only,
// and writes nothing but shared memory. Every kernel waits (whatever its blocks
// do afterwards), so "the one before" has itself waited for all earlier work.
// What the launch before writes is read by plain loads: a read-only load (__ldg)
// promises that nobody writes during the whole kernel, the part before its wait
// included, and the compiler may move it there. (Launches further back have
// completed when a kernel starts.) A kernel lets the next one be scheduled only
// once it has been released itself: let go before the wait, several waiting
// kernels pile up on the chip and the blocks of the working ones are placed
// unevenly (512x512 pair 219 us that way, 184 this way). These calls are chains
// of some thirty short dependent kernels, in which the launch latency is a large
// part: VGA single-level pair 133 -> 100 us, 512x512 at 8 layers 233 -> 184 us.
// The batched chain launches plainly.
template <class... P, class... A>
inline void launch_chained(void (*kernel)(P...), int grid, int block, int smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(block));
    cfg.dynamicSmemBytes = static_cast<std::size_t>(smem);
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);  // errors: launch_status()
}

__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

// Unique id of the current context (ids are never reused within a process); 0
// when there is none or it cannot be read.
unsigned long long current_context_id();

// Opts a kernel in to `most` bytes of dynamic shared memory in the current
// context; false if the device refuses. Once per context: the attribute belongs to
// the context it was set in, and a process may use several devices, or one again
// after a reset.
template <auto kKernel> bool enable_smem(int most) {
    static std::atomic<unsigned long long> done[64];  // by device: the context that has it
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return false;
    const unsigned long long context = dev < 64 ? current_context_id() : 0;
    if (context && done[dev].load(std::memory_order_relaxed) == context) return true;
    if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return false;
    if (dev < 64) done[dev].store(current_context_id(), std::memory_order_relaxed);  // the call may have made the context
    return true;
}

inline Status launch_status() {
    return cudaGetLastError() == cudaSuccess ? Status::OK : Status::CUDA_ERROR;
}

template <class T> inline T* at_offset(void* base, std::size_t offset) {
    return reinterpret_cast<T*>(static_cast<char*>(base) + offset);
}

inline bool aligned(const void* p, std::size_t a) {
    return (reinterpret_cast<std::uintptr_t>(p) % a) == 0;
}

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }

// Bump allocator over a workspace: every region starts on a 256-byte
// boundary; false on size_t overflow.
struct Layout {
    std::size_t cursor = 0;
    bool ok = true;
    std::size_t take(std::size_t count, std::size_t elem) {
        constexpr std::size_t kMax = ~std::size_t{0};
        if (!ok) return 0;
        if (cursor > kMax - (kWorkspaceAlign - 1)) { ok = false; return 0; }
        const std::size_t start = (cursor + kWorkspaceAlign - 1) / kWorkspaceAlign * kWorkspaceAlign;
        if (elem && count > (kMax - start) / elem) { ok = false; return 0; }
        cursor = start + count * elem;
        return start;
    }
};

}  // namespace stitch::b200
