// track_kernel.cu -- launches of the tracking kernel, and its instantiations
// for lattices without a lead block (KIND_SIMPLE); the other kinds are
// compiled beside it, in parallel.
#include <algorithm>

#include "track_kernel.cuh"

namespace stg {

STG_KIND(extern, KIND_PLAIN)
STG_KIND(extern, KIND_MAP)
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

// Threads per block where the caller gives none: the smallest block of which
// as many are resident on an SM (by shared memory) as the particles or the
// registers (512 threads) fill.  A scheduler with one warp runs an FP64
// instruction in 64 cycles, one of four busy ones in 76, and a second warp on
// a scheduler doubles its time, so small blocks, which spread evenly, win
// while all of them fit.  Measured, 32 / 64 / 128 threads: FODO ring, exact,
// 20,011 protons 0.62 / 0.65 / 0.78 ms, 40,000 0.79 / 0.83 / 0.94; beam-beam
// ring, fast, 40,000 1.14 / 1.19 / 1.32, 50,000 1.79 / 1.33 / 1.32, 65,536
// (64 / 128) 1.54 / 1.66; 2,000-element ring, exact, 131,072 3.28 / 3.33.
// Three stages of 8 KiB let nine blocks reside, four only six (131,072: 64
// threads 4.03 ms).
int default_track_threads(int64_t count, int n_chunks, int stages, int chunk_words)
{
    size_t const smem = track_smem_bytes(std::min(n_chunks, stages), chunk_words);
    int64_t const blocks = (int64_t)((228u << 10) / (smem + 1152u));
    int64_t const wanted = std::min<int64_t>((count + 151) / 152, 512);
    for (int threads : {32, 64})
        if (blocks * threads >= wanted) return threads;
    return 128;
}

int launch_track(const TrackParams &params, bool fast, int threads, int blocks_per_sm,
                 void *stream)
{
    TrackParams prm = params;
    int64_t const count = prm.live > 0 ? prm.live : prm.i1 - prm.i0;
    if (count <= 0) return 0;
    // a lattice that stays resident needs no more stages than it has chunks
    if (prm.n_chunks < prm.stages) prm.stages = prm.n_chunks;
    size_t const smem = track_smem_bytes(prm.stages, prm.chunk_words);
    if (threads <= 0)
        threads = default_track_threads(count, prm.n_chunks, prm.stages, prm.chunk_words);
    else if (threads > kMaxThreads || threads % 32 != 0)
        threads = kMaxThreads;
    unsigned const blocks = (unsigned)((count + threads - 1) / threads);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    bool const two = blocks_per_sm >= 2;
    switch (lattice_kind(prm.op_mask)) {
    case KIND_SIMPLE:
        return launch_kind<KIND_SIMPLE>(prm, fast, two, blocks, threads, smem, s);
    case KIND_PLAIN:
        return launch_kind<KIND_PLAIN>(prm, fast, two, blocks, threads, smem, s);
    case KIND_MAP:
        return launch_kind<KIND_MAP>(prm, fast, two, blocks, threads, smem, s);
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
    case KIND_MAP:
        return (int)batch_occupancy_kind<KIND_MAP>(fast, two, threads, smem, per_sm);
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
    case KIND_MAP:
        return launch_batch_kind<KIND_MAP>(b, s);
    default:
        return launch_batch_kind<KIND_FULL>(b, s);
    }
}

}  // namespace stg
