// fv_devbuf.hpp -- owned device buffers and the errors that the host code of the library throws (caught at
// the C ABI). Host code only; it includes no kernel.
#pragma once
#include <cuda_runtime_api.h>

#include <stdexcept>
#include <string>
#include <utility>

#include "ablate_fv.h"

namespace abl {

struct AblError : std::runtime_error {
    int code;
    AblError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define ABL_CUDA(call)                                                                                           \
    do {                                                                                                         \
        cudaError_t e_ = (call);                                                                                 \
        if (e_ != cudaSuccess) throw AblError(ABL_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() {
        if (p) cudaFree(p);
    }
    // After a failure the buffer is empty, n = 0 included: the callers that allocate on first use look at n, and
    // a later call must allocate again, not run on a null pointer. The error is taken off the runtime's record,
    // where the next launch check would find it.
    void alloc(size_t count) {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        if (count == 0) return;
        cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&p), count * sizeof(T));
        if (e != cudaSuccess) {
            p = nullptr;
            cudaGetLastError();
            throw AblError(e == cudaErrorMemoryAllocation ? ABL_ERR_OUT_OF_MEMORY : ABL_ERR_CUDA,
                           std::string("cudaMalloc: ") + cudaGetErrorString(e));
        }
        n = count;
    }
    // allocates unless the buffer has this size already (buffers made on first use)
    void ensure(size_t count) {
        if (n != count) alloc(count);
    }
    void swap(DevBuf& o) {
        std::swap(p, o.p);
        std::swap(n, o.n);
    }
    void upload(const T* h, size_t count) {
        alloc(count);
        if (count) ABL_CUDA(cudaMemcpy(p, h, count * sizeof(T), cudaMemcpyHostToDevice));
    }
    void zero() {
        if (n) ABL_CUDA(cudaMemset(p, 0, n * sizeof(T)));
    }
};

}  // namespace abl
