// Host program of test_pool_cpu.py: csrc/pool.cu over fakes of the CUDA calls it
// makes.  Prints one line per check that fails and exits with their number.
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../deconlib_b200/csrc/pool.cu"

static std::vector<std::string> calls;
static bool wait_ok = true, out_of_memory = false;
static int device = 0;
static uintptr_t next_ptr = 0x1000;
static void note(const char* name, const void* p = nullptr) {
    char b[64];
    snprintf(b, sizeof b, "%s %llx", name, (unsigned long long)(uintptr_t)p);
    calls.push_back(b);
}

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(uintptr_t)(0x10 + device); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { note("given back"); return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* q) { *p = (cudaMemPool_t)(uintptr_t)(0x20 + q->location.id); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { note("trim"); out_of_memory = false; return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) { a->device = ((uintptr_t)p >> 20) ? 1 : 0; return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t) {
    if (out_of_memory) return cudaErrorMemoryAllocation;
    *p = (void*)(next_ptr += 0x1000);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) { note(((uintptr_t)s & 0xf) == (unsigned)device ? "free" : "free on another device's stream", p); return cudaSuccess; }
// every way to wait for the device: refused together, as a lost context refuses them
cudaError_t cudaDeviceSynchronize() { if (!wait_ok) return cudaErrorStreamCaptureUnsupported; note("wait"); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) { *p = (void*)0x77; return cudaSuccess; }
cudaError_t cudaFree(void*) { if (!wait_ok) return cudaErrorStreamCaptureUnsupported; note("wait"); return cudaSuccess; }
}
namespace dk {
int fail(int code, const char*, ...) { return code; }
}

static int bad = 0;
static void expect(const char* what, const std::vector<std::string>& want) {
    if (calls != want) {
        ++bad;
        printf("%s:", what);
        for (auto& c : calls) printf(" [%s]", c.c_str());
        printf("\n");
    }
    calls.clear();
}

int main() {
    using namespace dk;
    void* const a = (void*)0xa00;
    void* const b = (void*)0xb00;
    void* const c = (void*)0xc00;
    void* const other = (void*)0x100a00;
    pool_free({nullptr, nullptr});
    expect("nothing to free", {});
    pool_free({a, nullptr, b});
    expect("one wait, then the buffers, then the pool's surplus", {"wait 0", "free a00", "free b00", "given back 0"});
    wait_ok = false;
    pool_free({a, b});
    expect("a refused wait frees nothing", {});
    wait_ok = true;
    pool_free({c});
    expect("the held buffers go after the next wait", {"wait 0", "free c00", "free a00", "free b00", "given back 0"});
    pool_free({c});
    expect("and only once", {"wait 0", "free c00", "given back 0"});
    wait_ok = false;
    pool_free({other});
    wait_ok = true;
    pool_free({a});
    expect("another device's buffers stay held", {"wait 0", "free a00", "given back 0"});
    pool_free({other});
    expect("until that device is waited for", {"wait 0", "free 100a00", "free 100a00", "given back 0"});
    if (device != 0) ++bad, printf("device not restored\n");
    wait_ok = false;
    pool_free({a});
    wait_ok = true;
    out_of_memory = true;
    void* p = nullptr;
    if (pool_alloc(&p, 64, "test") != DECON_OK || !p) ++bad, printf("allocation after a trim failed\n");
    expect("out of memory: held buffers and the pool's own go back", {"wait 0", "free a00", "given back 0", "trim 0", "given back 0"});
    return bad;
}
