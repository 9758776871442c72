// The CUDA context that calls of this thread run in. What the library keeps per
// device (kernel attributes, the address of a device array) belongs to a context:
// another one on the same device, after cudaDeviceReset for example, starts
// without it.
#include <cuda.h>

#include "common.cuh"

namespace {

using CtxGetCurrent = CUresult (*)(CUcontext*);
using CtxGetId = CUresult (*)(CUcontext, unsigned long long*);

struct DriverCalls {
    CtxGetCurrent get_current = nullptr;
    CtxGetId get_id = nullptr;
};

// cuCtxGetCurrent and cuCtxGetId through the runtime's driver entry points
// (the library links no libcuda); both null when the driver lacks them.
const DriverCalls& driver_calls() {
    static const DriverCalls calls = [] {
        DriverCalls c;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess && p)
            c.get_current = reinterpret_cast<CtxGetCurrent>(p);
        p = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess && p)
            c.get_id = reinterpret_cast<CtxGetId>(p);
        if (!c.get_current || !c.get_id) c = DriverCalls{};
        return c;
    }();
    return calls;
}

}  // namespace

namespace stitch::b200 {

unsigned long long current_context_id() {
    const DriverCalls& d = driver_calls();
    if (!d.get_current) return 0;
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (d.get_current(&ctx) != CUDA_SUCCESS || !ctx || d.get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

}  // namespace stitch::b200
