// Host-side check of the error word that a kernel sets when a bounded wait of
// its runs out (sync_checked and check_launch in
// lambda_vm_b200/csrc/common.cuh), compiled with g++ against a fake CUDA
// runtime: the word set while the stream is waited for fails that wait and
// every later launch and wait of the context, and no other context.
#include <stdio.h>

#include "../../lambda_vm_b200/csrc/common.cuh"

static volatile unsigned* g_set_on_sync = nullptr;  // the word a "kernel" sets before the wait returns
static cudaError_t g_sync_result = cudaSuccess;

cudaError_t cudaGetDevice(int* device) {
    *device = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    if (g_set_on_sync) *g_set_on_sync = 1;
    return g_sync_result;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
// page-locked memory: the calls that succeed, and the words held
static int g_host_calls_ok = 0, g_words = 0;
static unsigned g_word = 77;
cudaError_t cudaHostAlloc(void** host, size_t, unsigned) {
    if (g_host_calls_ok-- <= 0) return cudaErrorMemoryAllocation;
    ++g_words;
    *host = &g_word;
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** dev, void* host, unsigned) {
    if (g_host_calls_ok-- <= 0) return cudaErrorMemoryAllocation;
    *dev = host;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void*) {
    --g_words;
    return cudaSuccess;
}

namespace sg {
static thread_local std::string g_err;
void set_error(const std::string& msg) { g_err = msg; }
const char* last_error() { return g_err.c_str(); }
}  // namespace sg

#define EXPECT(cond)                                   \
    do {                                               \
        if (!(cond)) {                                 \
            printf("FAIL line %d: %s\n", __LINE__, #cond); \
            return 1;                                  \
        }                                              \
    } while (0)

int main() {
    unsigned wa = 0, wb = 0;
    sg::Ctx a, b, none;
    a.fault_host = &wa;
    b.fault_host = &wb;
    EXPECT(sg::check_launch(&a, "k") == SG_OK && sg::sync_checked(&a, nullptr, "x") == SG_OK);
    EXPECT(sg::sync_checked(&none, nullptr, "x") == SG_OK);  // a context without the word
    // the wait runs out after the launch was checked: the wait for the stream reports it
    EXPECT(sg::check_launch(&a, "k") == SG_OK);
    g_set_on_sync = &wa;
    EXPECT(sg::sync_checked(&a, nullptr, "x") == SG_ERR_CUDA);
    g_set_on_sync = nullptr;
    EXPECT(sg::sync_checked(&a, nullptr, "x") == SG_ERR_CUDA && sg::check_launch(&a, "k") == SG_ERR_CUDA);
    EXPECT(sg::check_launch(&b, "k") == SG_OK && sg::sync_checked(&b, nullptr, "x") == SG_OK);
    // the test hook: the third launch passes its own check and sets the word behind it
    b.fail_wait_after.store(3);
    for (int i = 0; i < 3; ++i) EXPECT(sg::check_launch(&b, "k") == SG_OK);
    EXPECT(sg::sync_checked(&b, nullptr, "x") == SG_ERR_CUDA);
    // no page-locked memory: a context without the word, and none left behind
    for (int calls = 0; calls < 3; ++calls) {
        sg::Ctx c;
        g_host_calls_ok = calls, g_words = 0;
        sg::alloc_fault_word(&c);
        EXPECT((c.fault_host != nullptr) == (calls == 2) && (c.fault_dev != nullptr) == (calls == 2));
        EXPECT(g_words == (calls == 2 ? 1 : 0) && (calls < 2 || *c.fault_host == 0));
        EXPECT(sg::check_launch(&c, "k") == SG_OK);
    }
    // a CUDA error of the wait itself is reported as before
    g_sync_result = cudaErrorInvalidDevice;
    EXPECT(sg::sync_checked(&none, nullptr, "prove") == SG_ERR_CUDA);
    EXPECT(std::string(sg::last_error()) == "prove: fake");
    printf("ok\n");
    return 0;
}
