// Host-only check that every call works on each device of one process, not on
// the first alone: the built objects are linked to the CUDA runtime below, which
// keeps kernel attributes per device, as the real one does, and refuses a launch
// with more than 48 KB of dynamic shared memory of a kernel that was not opted
// in on the current device; a reset takes the attributes away. It also checks the
// blocks of a batch whose jobs have far more candidates than keys may be there.
// Nothing runs on a GPU. Built and run by tests/test_multi_device.py.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <utility>
#include <vector>

#include "stitch_b200.h"

namespace {

int device = 0, launches = 0, refused = 0, set = 0;
bool with_ids = false;                // whether the driver tells contexts apart
unsigned long long context[8] = {1, 2, 3, 4, 5, 6, 7, 8};
bool refuse_attributes = false;
std::map<std::pair<int, const void*>, std::size_t> opted;
cudaError_t last = cudaSuccess;

unsigned rank_blocks = 0;  // most blocks of 512 threads, the ranking's, of a launch

cudaError_t launch(const void* kernel, dim3 grid, dim3 block, std::size_t smem) {
    if (block.x == 512 && grid.x > rank_blocks) rank_blocks = grid.x;
    const auto it = opted.find({device, kernel});
    const std::size_t limit = it == opted.end() ? 48 * 1024 : it->second;
    ++launches;
    if (smem <= limit) return cudaSuccess;
    ++refused;
    return last = cudaErrorInvalidValue;
}

struct Call {
    dim3 grid, block;
    std::size_t smem = 0;
    void* stream = nullptr;
} pending;

void* host_memory(std::size_t n) { return std::aligned_alloc(256, (n + 255) / 256 * 256); }

}  // namespace

extern "C" {
void** __cudaRegisterFatBinary(void*) {
    static void* handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, std::size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, std::size_t smem, void* s) {
    pending = {g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, std::size_t* smem, void* s) {
    *g = pending.grid;
    *b = pending.block;
    *smem = pending.smem;
    *static_cast<void**>(s) = pending.stream;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return device = d, cudaSuccess; }
cudaError_t cudaGetLastError() { return std::exchange(last, cudaSuccess); }
cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute a, int value) {
    if (refuse_attributes) return last = cudaErrorInvalidValue;
    ++set;
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) opted[{device, kernel}] = static_cast<std::size_t>(value);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* kernel, dim3 grid, dim3 block, void**, std::size_t smem, cudaStream_t) {
    return launch(kernel, grid, block, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* kernel, void**) {
    return launch(kernel, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaMemcpyAsync(void*, const void*, std::size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void*, std::size_t, const void*, std::size_t, std::size_t, std::size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, std::size_t n, std::size_t, cudaMemcpyKind) { return std::memset(d, 0, n), cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, std::size_t, std::size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, std::size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, std::size_t n) { return *p = host_memory(n), cudaSuccess; }
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, std::size_t n, unsigned) { return *p = host_memory(n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return *p = &device, cudaSuccess; }
CUresult current(CUcontext* c) { return *c = reinterpret_cast<CUcontext>(&context[device]), CUDA_SUCCESS; }
CUresult context_id(CUcontext c, unsigned long long* id) { return *id = *reinterpret_cast<unsigned long long*>(c), CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *p = reinterpret_cast<void*>(!std::strcmp(name, "cuCtxGetCurrent") ? reinterpret_cast<void (*)()>(current) : reinterpret_cast<void (*)()>(context_id));
    *q = cudaDriverEntryPointSuccess;
    return with_ids ? cudaSuccess : cudaErrorNotSupported;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { return *s = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}

namespace {

constexpr int kCap = 9000;  // rows of every buffer

struct Buffers {
    void* ws = host_memory(64 << 20);
    float* f = static_cast<float*>(host_memory(sizeof(float) * kCap));
    int* i = static_cast<int*>(host_memory(sizeof(int) * kCap));
    void* desc = host_memory(32 * kCap);
    unsigned char* bytes = static_cast<unsigned char*>(host_memory(640 * 480));
};

stitch_pair_desc pair(const Buffers& b, int k, int hypotheses, int levels) {
    stitch_pair_desc d{};
    d.image_a = d.image_b = stitch_image_view{b.bytes, 640, 480, 640, 1};
    d.s2 = stitch_s2_config{20, k, 0.04f};
    d.s4.ratio_threshold = 0.8f;
    d.s5 = stitch_s5_config{hypotheses, 0, 64, 1, 3.0, 7, 1};
    d.pyramid = stitch_pyramid_config{levels, 1.2f};
    return d;
}

int estimate(const Buffers& b, int capacity, int hypotheses) {
    const stitch_keypoints kp{b.f, b.f, b.f, capacity, b.i};
    const stitch_matches m{b.i, b.i, b.f, capacity, b.i};
    stitch_scale_info si{};
    stitch_make_scale_info(640, 480, 1.0, &si);
    const stitch_s5_config c{hypotheses, 0, 64, 1, 3.0, 7, 1};
    stitch_homography_result out{};
    return stitch_s5_estimate(&kp, &kp, &m, &si, &si, &c, b.bytes, &out, b.ws, 64 << 20, nullptr);
}

int detect_and_match(const Buffers& b, int k) {
    const stitch_image_view im{b.bytes, 640, 480, 640, 1};
    const stitch_s2_config c2{20, k, 0.04f};
    const stitch_keypoints kp{b.f, b.f, b.f, k, b.i};
    const stitch_descriptors d{0, 32, 32, b.desc};
    const stitch_pyramid_config p{8, 1.2f};
    stitch_s4_config c4{};
    c4.ratio_threshold = 0.8;
    c4.cross_check = 1;
    const stitch_matches m{b.i, b.i, b.f, k, b.i};
    int st = stitch_s2_detect(&im, &c2, &kp, b.ws, 64 << 20, nullptr);
    if (!st) st = stitch_s3_describe(&im, &kp, &d, b.ws, 64 << 20, nullptr);
    if (!st) st = stitch_pyramid_detect_describe(&im, &c2, &p, &kp, &d, b.ws, 64 << 20, nullptr);
    for (int kind = 0; !st && kind <= 4; ++kind) {
        st = stitch_s4_set_matcher(kind);
        if (!st) st = stitch_s4_match(&kp, &d, &kp, &d, &c4, &m, b.ws, 64 << 20, nullptr);
    }
    stitch_s4_set_matcher(1);
    return st;
}

int batch(const Buffers& b, int k, int levels, const stitch_batch_tuning* tuning, int copies = 1) {
    std::vector<stitch_pair_desc> pairs(copies, pair(b, k, 2000, levels));
    pairs.push_back(pair(b, 500, 500, levels));
    stitch_batch* plan = nullptr;
    std::size_t bytes = 0;
    int bad = -1;
    int st = stitch_batch_create_tuned(static_cast<int>(pairs.size()), pairs.data(), tuning, &plan, &bytes, &bad);
    if (st) return st;
    void* ws = host_memory(bytes);
    st = stitch_batch_enqueue(plan, ws, bytes, nullptr, nullptr);
    std::free(ws);
    stitch_batch_destroy(plan);
    return st;
}

}  // namespace

int main(int argc, char**) {
    const Buffers b;
    with_ids = argc > 1;
    for (int d = 0; d < 3; ++d) {
        cudaSetDevice(d);
        for (const int k : {100, 2000, 8193}) {
            for (const int r : {500, 2000, 4000, 8000})
                if (const int st = estimate(b, k, r)) return std::printf("device %d: estimate of %d: status %d\n", d, k, st), 1;
            if (const int st = detect_and_match(b, k)) return std::printf("device %d: stages at K = %d: status %d\n", d, k, st), 1;
            for (const int hpw : {0, 4, 8, 16, 32})
                for (const int levels : {1, 8}) {
                    const stitch_batch_tuning t{0, 0, 0, hpw, 0};
                    if (const int st = batch(b, k, levels, &t))
                        return std::printf("device %d: batch of K = %d, %d levels: status %d\n", d, k, levels, st), 1;
                }
        }
        if (refused) return std::printf("device %d: %d launches refused\n", d, refused), 1;
    }
    // a reset: another context without the attributes; and, the contexts known, no attribute is set twice
    cudaSetDevice(1);
    opted.clear();
    context[1] = 100;
    {
        if (const int st = estimate(b, 8193, 2000)) return std::printf("after a reset: estimate: status %d\n", st), 1;
        if (const int st = detect_and_match(b, 8193)) return std::printf("after a reset: stages: status %d\n", st), 1;
        if (const int st = batch(b, 8193, 8, nullptr)) return std::printf("after a reset: batch: status %d\n", st), 1;
    }
    const int before_again = set;
    estimate(b, 8193, 2000), detect_and_match(b, 8193), batch(b, 8193, 8, nullptr);
    if (with_ids && set != before_again) return std::printf("attributes set again\n"), 1;
    // 32 pairs of 2 x 40000 candidates: a block per 32 of them would be 80,000 blocks
    rank_blocks = 0;
    if (const int st = batch(b, 20000, 1, nullptr, 32)) return std::printf("large batch: status %d\n", st), 1;
    if (rank_blocks == 0 || rank_blocks > 2000) return std::printf("%u blocks of the ranking\n", rank_blocks), 1;
    // a device that refuses the attribute: an error, and no launch that would fail
    cudaSetDevice(3);
    refuse_attributes = true;
    const int before = launches;
    if (estimate(b, 2000, 500) == 0 || batch(b, 2000, 1, nullptr) == 0) return std::printf("refusal not reported\n"), 1;
    if (launches != before) return std::printf("launched without the attribute\n"), 1;
    std::printf("devices ok: %d launches\n", launches);
    return 0;
}
