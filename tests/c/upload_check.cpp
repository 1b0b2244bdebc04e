// Runs the scene loader (csrc/scene.cpp) on a CUDA runtime of host memory whose
// fills and copies to the device do no more than they promise: the bytes are
// taken at the call and arrive when the stream is waited for.  Arguments: an
// .rle4 file, and the number of the wait that fails (0: none).  Prints the
// loader's status, the operations still on the way when it returned, and
// whether it returned a scene.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "rle_internal.h"

namespace {
struct Op {
    void* to;
    std::vector<char> bytes;
};
std::vector<Op> on_the_way;
int waits = 0, waits_fail_at = 0;
}  // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    if (++waits == waits_fail_at) return cudaErrorUnknown;
    for (const Op& o : on_the_way) std::memcpy(o.to, o.bytes.data(), o.bytes.size());
    on_the_way.clear();
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaStreamSynchronize(nullptr); }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::malloc(n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) {
    cudaStreamSynchronize(nullptr);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind kind) {
    if (kind == cudaMemcpyHostToDevice) {
        on_the_way.push_back({to, std::vector<char>(static_cast<const char*>(from), static_cast<const char*>(from) + n)});
        return cudaSuccess;
    }
    const cudaError_t e = cudaStreamSynchronize(nullptr);  // copies to the host wait
    if (e == cudaSuccess) std::memcpy(to, from, n);
    return e;
}
cudaError_t cudaMemset(void* to, int v, size_t n) {
    on_the_way.push_back({to, std::vector<char>(n, static_cast<char>(v))});
    return cudaSuccess;
}
}

int main(int argc, char** argv) {
    if (argc < 3) return 2;
    waits_fail_at = std::atoi(argv[2]);
    rle_scene* s = nullptr;
    const rle_status st = rle_scene_load_file(argv[1], 0, &s);
    std::printf("%d %zu %d\n", static_cast<int>(st), on_the_way.size(), s != nullptr);
    if (s) rle_scene_free(s);
    return 0;
}
