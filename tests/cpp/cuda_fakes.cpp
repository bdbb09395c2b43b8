// Stand-ins for two CUDA runtime calls, linked in front of the real ones (-Wl,--wrap): a stream-ordered
// allocation that fails as out of memory at chosen sizes, and a copy from pageable host memory that
// reads its source when the stream reaches the copy, as the runtime's documentation allows.
#include <cuda_runtime.h>

#include <chrono>
#include <cstring>
#include <thread>

extern "C" {
cudaError_t __real_cudaMallocAsync(void **, size_t, cudaStream_t);
cudaError_t __real_cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t);

static size_t g_fail[4];
static int g_failed, g_late, g_lates;

void fake_fail_allocations(size_t a, size_t b) {
    g_fail[0] = a;
    g_fail[1] = b;
    g_failed = 0;
}
int fake_failed() { return g_failed; }
void fake_late_copies(int on) {
    g_late = on;
    g_lates = 0;
}
int fake_lates() { return g_lates; }

cudaError_t __wrap_cudaMallocAsync(void **p, size_t bytes, cudaStream_t s) {
    if (bytes && (bytes == g_fail[0] || bytes == g_fail[1])) {
        ++g_failed;
        return cudaErrorMemoryAllocation;
    }
    return __real_cudaMallocAsync(p, bytes, s);
}

struct Late {
    const void *src;
    void *staging;
    size_t bytes;
};
static void read_late(void *arg) {
    Late *l = (Late *)arg;
    std::this_thread::sleep_for(std::chrono::milliseconds(2));
    std::memcpy(l->staging, l->src, l->bytes);
    delete l;  // the staging buffer stays: a test makes few copies
}

cudaError_t __wrap_cudaMemcpyAsync(void *dst, const void *src, size_t bytes, cudaMemcpyKind kind, cudaStream_t s) {
    if (!g_late || kind != cudaMemcpyHostToDevice || !bytes) return __real_cudaMemcpyAsync(dst, src, bytes, kind, s);
    Late *l = new Late{src, nullptr, bytes};
    cudaError_t e = cudaHostAlloc(&l->staging, bytes, cudaHostAllocDefault);
    void *staging = l->staging;
    if (e == cudaSuccess) e = cudaLaunchHostFunc(s, read_late, l);
    if (e != cudaSuccess) return e;
    ++g_lates;
    return __real_cudaMemcpyAsync(dst, staging, bytes, kind, s);
}
}
