// What surrounds the layers of a step: rows gathered from tables (token embeddings, rotary tables) and the greedy token of every row
// of logits.
#include <assert.h>
#include <cooperative_groups.h>
#include <utility>

#include "typed_io.cuh"

namespace sllm {

namespace cg = cooperative_groups;

// Row t of out_a is row idx[t] + offset of table_a, row t of out_b the same row of table_b, or zeros without a table_b.  One CTA per row;
// rows are moved as pieces of 16, 4 or 2 bytes (P), whichever their lengths and addresses allow.  Bound: one launch and one dependent
// load.  Measured on B200, 16 rows: an embedding of 4096 entries with a zeroed residual 2 us, both rotary tables 2 us; the index
// selections and fills of the tensor library that this replaces took 13, 13 and 2 us.
template <typename P>
__global__ void __launch_bounds__(256) gather_rows_kernel(const int* __restrict__ idx, int offset, int64_t table_rows,
                                                          const P* __restrict__ table_a, P* __restrict__ out_a, int na,
                                                          const P* __restrict__ table_b, P* __restrict__ out_b, int nb) {
    wait_previous();
    launch_next();
    idx = after_wait(idx); table_a = after_wait(table_a); table_b = after_wait(table_b);
    const int64_t t = blockIdx.x, r = (int64_t)idx[t] + offset;
    assert(r >= 0 && r < table_rows);
    for (int i = threadIdx.x; i < na; i += blockDim.x) out_a[t * na + i] = table_a[r * na + i];
    for (int i = threadIdx.x; i < nb; i += blockDim.x) out_b[t * nb + i] = table_b != nullptr ? table_b[r * nb + i] : P{};
}

template <typename P>
static void launch_gather(const int* idx, int offset, int64_t table_rows, const void* ta, void* oa, int64_t bytes_a, const void* tb, void* ob,
                          int64_t bytes_b, int64_t n, cudaStream_t s) {
    const int na = (int)(bytes_a / (int64_t)sizeof(P)), nb = (int)(bytes_b / (int64_t)sizeof(P)), most = na > nb ? na : nb;
    launch_early(gather_rows_kernel<P>, (unsigned)n, most >= 256 ? 256 : (most + 31) / 32 * 32, 0, s, idx, offset, table_rows, (const P*)ta, (P*)oa, na,
                 (const P*)tb, (P*)ob, nb);
}

// The greater of two (value, index) pairs: NaN above everything, the smaller index among equals.
__device__ __forceinline__ bool above(float v, int i, float w, int j) {
    if (isnan(v) || isnan(w)) return isnan(v) && (!isnan(w) || i < j);
    return v > w || (v == w && i < j);
}

// Eight CTAs (a cluster) per row, each over every eighth run of 256 pieces of VEC entries; the eight results meet in the first CTA's shared
// memory, which may be written once that CTA is known to run: all arrive at the cluster's barrier as they start, and wait at it behind
// their loads.  One launch whatever the number of rows: a row has eight CTAs' loads in flight, 256 rows fill the GPU.  Bound: the bytes
// of the logits (in L2 behind the head's product), below about 32 rows one load's latency per run.  Measured on B200, 128256 entries of
// 16 bits, us, this / the tensor library's reduction: 16 rows 6.4 / 26, 64 rows 12 / 26, 128 rows 18, 256 rows 31 / 37.
constexpr int AM_CTAS = 8, AM_THREADS = 256, AM_RUNS = 4;
template <typename T, int VEC>
__global__ void __cluster_dims__(AM_CTAS, 1, 1) __launch_bounds__(AM_THREADS) argmax_rows_kernel(const T* __restrict__ x, int64_t stride, int n,
                                                                                                int64_t* __restrict__ out) {
    struct alignas(VEC * sizeof(T)) Piece { T e[VEC]; };
    __shared__ float wv[AM_THREADS / 32], cv[AM_CTAS];
    __shared__ int wi[AM_THREADS / 32], ci[AM_CTAS];
    cg::cluster_group cluster = cg::this_cluster();
    auto here = cluster.barrier_arrive();                            // this CTA has started
    wait_previous();
    launch_next();
    x = after_wait(x);
    const int rank = (int)cluster.block_rank(), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row = blockIdx.x / AM_CTAS;
    const T* p = x + row * stride;
    const int pieces = n / VEC, step = AM_CTAS * AM_THREADS;
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int i0 = rank * AM_THREADS + threadIdx.x; i0 < pieces; i0 += step * AM_RUNS) {
        Piece v[AM_RUNS];
#pragma unroll
        for (int u = 0; u < AM_RUNS; u++)
            if (i0 + u * step < pieces) v[u] = reinterpret_cast<const Piece*>(p)[i0 + u * step];
#pragma unroll
        for (int u = 0; u < AM_RUNS; u++)
            if (i0 + u * step < pieces) {
#pragma unroll
                for (int e = 0; e < VEC; e++) {
                    const float f = ldf(&v[u].e[e]);
                    const int i = (i0 + u * step) * VEC + e;
                    if (above(f, i, best, at)) { best = f; at = i; }
                }
            }
    }
    auto across = [&](float& v, int& i, int width) {
        for (int o = width / 2; o > 0; o >>= 1) {
            const float w = __shfl_xor_sync(0xffffffffu, v, o);
            const int j = __shfl_xor_sync(0xffffffffu, i, o);
            if (above(w, j, v, i)) { v = w; i = j; }
        }
    };
    across(best, at, 32);
    if (lane == 0) { wv[warp] = best; wi[warp] = at; }
    cluster.barrier_wait(std::move(here));                           // the first CTA has: its shared memory may be written
    __syncthreads();
    if (warp == 0) {
        best = wv[lane & 7]; at = wi[lane & 7];
        across(best, at, 8);
        if (lane == 0) {
            *cluster.map_shared_rank(&cv[rank], 0) = best;
            *cluster.map_shared_rank(&ci[rank], 0) = at;
        }
    }
    cluster.sync();
    if (rank == 0 && warp == 0) {
        best = cv[lane & 7]; at = ci[lane & 7];
        across(best, at, 8);
        if (lane == 0) out[row] = at;
    }
}

}  // namespace sllm

using namespace sllm;

extern "C" {

int sllm_gather_rows(const void* idx, int offset, int64_t num_rows, int64_t table_rows, const void* table_a, void* out_a, int64_t row_bytes_a,
                     const void* table_b, void* out_b, int64_t row_bytes_b, sllm_stream_t stream) {
    SLLM_REQUIRE(num_rows >= 0 && table_rows >= 0 && row_bytes_a > 0 && row_bytes_b >= 0 && row_bytes_a % 2 == 0 && row_bytes_b % 2 == 0 &&
                 row_bytes_a < (1ll << 31) && row_bytes_b < (1ll << 31), "gather_rows: bad shape (%lld rows of %lld and %lld bytes)",
                 (long long)num_rows, (long long)row_bytes_a, (long long)row_bytes_b);
    if (num_rows == 0) return 0;
    SLLM_REQUIRE(idx && table_a && out_a && (row_bytes_b == 0 || out_b), "gather_rows: null pointer");
    const uint64_t all = (uintptr_t)table_a | (uintptr_t)out_a | (uintptr_t)table_b | (uintptr_t)out_b | (uint64_t)row_bytes_a | (uint64_t)row_bytes_b;
    SLLM_REQUIRE(all % 2 == 0, "gather_rows: addresses must be even");
    cudaStream_t s = (cudaStream_t)stream;
    if (all % 16 == 0) launch_gather<uint4>((const int*)idx, offset, table_rows, table_a, out_a, row_bytes_a, table_b, out_b, row_bytes_b, num_rows, s);
    else if (all % 4 == 0) launch_gather<uint32_t>((const int*)idx, offset, table_rows, table_a, out_a, row_bytes_a, table_b, out_b, row_bytes_b, num_rows, s);
    else launch_gather<unsigned short>((const int*)idx, offset, table_rows, table_a, out_a, row_bytes_a, table_b, out_b, row_bytes_b, num_rows, s);
    return check_launch("gather_rows");
}

int sllm_argmax_rows(const void* x, int64_t row_stride, int64_t num_rows, int64_t n, void* out, sllm_dtype_t dtype, sllm_stream_t stream) {
    SLLM_REQUIRE(num_rows >= 0 && n > 0 && n < (1ll << 30) && row_stride >= 0 && num_rows < (1ll << 28), "argmax_rows: bad shape (%lld rows of %lld)", (long long)num_rows, (long long)n);
    if (num_rows == 0) return 0;
    SLLM_REQUIRE(x && out, "argmax_rows: null pointer");
    const unsigned grid = (unsigned)(num_rows * AM_CTAS);
    cudaStream_t s = (cudaStream_t)stream;
    SLLM_DISPATCH_DTYPE_F32(dtype, {
        constexpr int W = 16 / (int)sizeof(T);
        if (n % W == 0 && row_stride % W == 0 && ((uintptr_t)x & 15) == 0)
            launch_early(argmax_rows_kernel<T, W>, grid, AM_THREADS, 0, s, (const T*)x, row_stride, (int)n, (int64_t*)out);
        else
            launch_early(argmax_rows_kernel<T, 1>, grid, AM_THREADS, 0, s, (const T*)x, row_stride, (int)n, (int64_t*)out);
    });
    return check_launch("argmax_rows");
}

}  // extern "C"
