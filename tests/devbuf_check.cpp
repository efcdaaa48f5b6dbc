// Host-side check of the owned device buffers (ablate_b200/csrc/fv_devbuf.hpp), compiled with g++ by
// tests/test_devbuf.py against the stand-ins of the CUDA runtime below: what a buffer claims after an
// allocation failed, and that the caller's next attempt allocates. Prints "ok" or the failed expectation.
#include <cstdio>
#include <cstdlib>

#include "fv_devbuf.hpp"

static int g_fail = 0;   // the next cudaMalloc calls that fail
static int g_live = 0;   // allocations held
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    if (g_fail > 0) {
        g_fail--;
        return g_last = cudaErrorMemoryAllocation;
    }
    *p = std::malloc(n);
    g_live++;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    g_live--;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
}

#define EXPECT(c)                                    \
    if (!(c)) {                                      \
        std::printf("line %d: %s\n", __LINE__, #c);  \
        return 1;                                    \
    }

static int code_of(abl::DevBuf<double>& b, size_t n) {
    try {
        b.ensure(n);
    } catch (const abl::AblError& e) {
        return e.code;
    }
    return ABL_OK;
}

int main() {
    {
        abl::DevBuf<double> b;
        g_fail = 1;
        EXPECT(code_of(b, 100) == ABL_ERR_OUT_OF_MEMORY);
        EXPECT(b.p == nullptr && b.n == 0);          // a first-use check looks at n
        EXPECT(cudaGetLastError() == cudaSuccess);   // a launch check would report it for a launch
        EXPECT(code_of(b, 100) == ABL_OK && b.p != nullptr && b.n == 100);
        double* const p = b.p;
        EXPECT(code_of(b, 100) == ABL_OK && b.p == p);
        g_fail = 1;
        EXPECT(code_of(b, 200) == ABL_ERR_OUT_OF_MEMORY);
        EXPECT(b.p == nullptr && b.n == 0);
        EXPECT(code_of(b, 0) == ABL_OK && b.p == nullptr && b.n == 0);
        abl::DevBuf<double> c;
        EXPECT(code_of(c, 7) == ABL_OK);
        b.swap(c);
        EXPECT(b.n == 7 && b.p != nullptr && c.n == 0 && c.p == nullptr);
    }
    EXPECT(g_live == 0);
    std::printf("ok\n");
    return 0;
}
