// track_kernel.cu -- launches of the tracking kernel, and its instantiations
// for lattices without a lead block (KIND_SIMPLE); the other kinds are
// compiled beside it, in parallel.
#include "track_kernel.cuh"

namespace stg {

STG_KIND(extern, KIND_PLAIN)
STG_KIND(extern, KIND_FULL)
STG_KIND(, KIND_SIMPLE)

namespace {
__global__ void __launch_bounds__(256) exp_fast_kernel(const double *x, double *y, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        y[i] = exp_fast(x[i]);
}
}  // namespace

namespace {
__global__ void __launch_bounds__(256) rcp_fast_kernel(const double *x, double *y, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        y[i] = rcp_fast(x[i]);
}
}  // namespace

int launch_rcp_fast(const double *x, double *y, int64_t n, void *stream)
{
    if (n <= 0) return 0;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    rcp_fast_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, y, n);
    return (int)cudaGetLastError();
}

int launch_exp_fast(const double *x, double *y, int64_t n, void *stream)
{
    if (n <= 0) return 0;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 152 * 32) blocks = 152 * 32;
    exp_fast_kernel<<<(unsigned)blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(x, y, n);
    return (int)cudaGetLastError();
}

size_t track_smem_bytes(int stages, int chunk_words)
{
    return (size_t)(16 + (size_t)stages * chunk_words) * sizeof(uint64_t);
}

int launch_track(const TrackParams &prm, bool fast, int threads, int blocks_per_sm, void *stream)
{
    int64_t const count = prm.i1 - prm.i0;
    if (count <= 0) return 0;
    if (threads <= 0 || threads > kMaxThreads || threads % 32 != 0) threads = kMaxThreads;
    unsigned const blocks = (unsigned)((count + threads - 1) / threads);
    size_t const smem = track_smem_bytes(prm.stages, prm.chunk_words);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    bool const two = blocks_per_sm >= 2;
    switch (lattice_kind(prm.op_mask)) {
    case KIND_SIMPLE:
        return launch_kind<KIND_SIMPLE>(prm, fast, two, blocks, threads, smem, s);
    case KIND_PLAIN:
        return launch_kind<KIND_PLAIN>(prm, fast, two, blocks, threads, smem, s);
    default:
        return launch_kind<KIND_FULL>(prm, fast, two, blocks, threads, smem, s);
    }
}

int batch_ctas_per_sm(bool fast, LatticeKind kind, int threads, int blocks_per_sm, size_t smem,
                      int *per_sm)
{
    bool const two = blocks_per_sm >= 2;
    switch (kind) {
    case KIND_SIMPLE:
        return (int)batch_occupancy_kind<KIND_SIMPLE>(fast, two, threads, smem, per_sm);
    case KIND_PLAIN:
        return (int)batch_occupancy_kind<KIND_PLAIN>(fast, two, threads, smem, per_sm);
    default:
        return (int)batch_occupancy_kind<KIND_FULL>(fast, two, threads, smem, per_sm);
    }
}

int launch_batch(const BatchLaunch &b, void *stream)
{
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (b.kind) {
    case KIND_SIMPLE:
        return launch_batch_kind<KIND_SIMPLE>(b, s);
    case KIND_PLAIN:
        return launch_batch_kind<KIND_PLAIN>(b, s);
    default:
        return launch_batch_kind<KIND_FULL>(b, s);
    }
}

}  // namespace stg
