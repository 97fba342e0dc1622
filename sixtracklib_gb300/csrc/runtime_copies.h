// runtime_copies.h -- the CUDA runtime's copies for column_copy.h.
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "column_copy.h"
#include "common.h"

namespace stg {

// On `stream`; null copies as cudaMemcpy does.
struct RuntimeCopies {
    cudaMemcpyKind kind;
    cudaStream_t stream;
    const char *what;
    bool ok(cudaError_t e) const
    {
        if (e == cudaSuccess) return true;
        set_error(std::string(what) + ": " + cudaGetErrorString(e));
        return false;
    }
    bool copy(void *to, const void *from, size_t bytes)
    {
        return ok(stream ? cudaMemcpyAsync(to, from, bytes, kind, stream)
                         : cudaMemcpy(to, from, bytes, kind));
    }
    bool copy2d(void *to, size_t tp, const void *from, size_t fp, size_t width, size_t rows)
    {
        return ok(stream ? cudaMemcpy2DAsync(to, tp, from, fp, width, rows, kind, stream)
                         : cudaMemcpy2D(to, tp, from, fp, width, rows, kind));
    }
    bool wait() { return ok(cudaStreamSynchronize(stream)); }
};

// Tables from host vectors, in device memory on return.
inline bool upload(std::initializer_list<BlockCopy> blocks, const char *what)
{
    RuntimeCopies api{cudaMemcpyHostToDevice, nullptr, what};
    return copy_blocks(api, blocks);
}

}  // namespace stg
