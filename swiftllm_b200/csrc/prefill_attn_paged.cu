// Chunked ("prefix-aware") prefill attention: the queries of a prompt CHUNK attend to the whole prefix + chunk through
// the paged KV cache.  The reference's forward cannot express a partial prompt (its prefill attention,
// swiftllm/worker/kernels/prefill_attn.py:102-139 / transformer_layer.py:86-96, only ever sees the packed k/v of the
// batch), which is what SARATHI-style piggybacking needs.  Definition = the one that makes
// a prompt processed in chunks equal to the same prompt processed at once (oracle/kernels.py:
// prefix_prefill_attention_exact).  Both generations of the prefill kernel are instantiated with PAGED = true:
//   gen 2 (prefill_attn_tc_kernel.cuh): tcgen05 + TMA page gather, head_dim 128, block_size 16
//   gen 1 (prefill_attn_kernel.cuh):    cp.async page gather + mma.sync, head_dim 64 / 128, any block_size
// Roofline: tensor-bound; FLOPs = 4 * nq * D * sum_i (prefix_i * L_i + L_i (L_i + 1) / 2).
#include <stdlib.h>

#include "prefill_attn_kernel.cuh"
#include "prefill_attn_tc_kernel.cuh"

namespace sllm {

template <typename T, int D>
static int launch_prefill_paged(const void* q, const void* k_cache, const void* v_cache, void* o, const int32_t* start_locs,
                                const int32_t* chunk_lens, float scale, int num_seqs, int max_chunk_len, int nq, int nkv,
                                int64_t qs, const PfPagedKV& pk, cudaStream_t stream) {
    const size_t smem = (size_t)PF_BQ * D * 2 + 2 * 2 * (size_t)PF_BK * D * 2;
    static unsigned long long configured = 0;
    if (first_use_on_this_device(configured)) {
        cudaFuncSetAttribute(prefill_attn_kernel<T, D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    dim3 grid(cdiv(max_chunk_len, PF_BQ), nq, num_seqs);
    prefill_attn_kernel<T, D, true><<<grid, PF_THREADS, smem, stream>>>((const T*)q, (const T*)k_cache, (const T*)v_cache, (T*)o,
                                                                       start_locs, chunk_lens, scale * 1.4426950408889634f, nq,
                                                                       nkv, qs, 0, 0, pk);
    return check_launch("prefill_attention_paged");
}

// One warp per (row of sequence blockIdx.y, head), four entries a lane: the splits' rows on their common maximum.  A split that saw no key
// of the row has the sum 0 and may have written no O (a sum that is NaN belongs to keys that it saw).  Rows of no sequence are left alone.
template <typename T>
__global__ void __launch_bounds__(256) prefill_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                            T* __restrict__ o, const int32_t* __restrict__ start_locs,
                                                            const int32_t* __restrict__ seq_lens, int nq, int64_t units, int nsplit) {
    wait_previous();
    launch_next();
    part_o = after_wait(part_o); part_ml = after_wait(part_ml); start_locs = after_wait(start_locs); seq_lens = after_wait(seq_lens);
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int start = start_locs[blockIdx.y], len = seq_lens[blockIdx.y];
    if (i >= (int64_t)len * nq) return;
    const int64_t u = (int64_t)start * nq + i;
    float M = -INFINITY, L = 0.f;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int z = 0; z < nsplit; z += 2) {            // two splits' loads in flight, none waits for another
        float2 ml[2];
        float4 v[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int64_t at = min(z + k, nsplit - 1) * units + u;
            ml[k] = *reinterpret_cast<const float2*>(part_ml + 2 * at);
            v[k] = *reinterpret_cast<const float4*>(part_o + at * PT_D + 4 * lane);
        }
        if (z + 1 == nsplit) ml[1] = make_float2(-INFINITY, 0.f);
        const float m = fmaxf(M, fmaxf(ml[0].x, ml[1].x)), keep = M == m ? 1.f : exp2f(M - m);
        M = m; L *= keep;
        a.x *= keep; a.y *= keep; a.z *= keep; a.w *= keep;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (ml[k].y == 0.f) continue;            // (its O is whatever lay there)
            const float f = exp2f(ml[k].x - m);
            L += f * ml[k].y;
            a.x += f * v[k].x; a.y += f * v[k].y; a.z += f * v[k].z; a.w += f * v[k].w;
        }
    }
    const float inv = 1.f / L;
    typename Traits<T>::T2 lo = Traits<T>::from_f2(make_float2(a.x * inv, a.y * inv)), hi = Traits<T>::from_f2(make_float2(a.z * inv, a.w * inv));
    *reinterpret_cast<uint2*>(o + u * PT_D + 4 * lane) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}

static bool tc_prefill_paged_supported(int head_dim, int block_size, int64_t num_tokens, int64_t cache_rows) {
    return head_dim == PT_D && block_size == PT_PAGE && num_tokens > 0 && num_tokens < (1LL << 31) &&
           cache_rows < (1LL << 31) && get_tensor_map_encoder() != nullptr;      // TMA coordinates are int32
}

static int launch_prefill_paged_tc(const void* q, const void* k_cache, const void* v_cache, void* o, const int32_t* start_locs,
                                   const int32_t* chunk_lens, float scale_log2e, int num_seqs, int max_chunk_len,
                                   int64_t num_tokens, int nq, int nkv, int64_t qs, int64_t cache_rows, const PtPaged& pg,
                                   sllm_dtype_t dtype, cudaStream_t stream) {
    PtParams p;
    p.o = o; p.start_locs = start_locs; p.seq_lens = chunk_lens; p.scale_log2e = scale_log2e; p.nq = nq; p.nkv = nkv;
    bool many;
    const dim3 grid = pt_grid(p, num_seqs, max_chunk_len, num_tokens, pg.nsplit, true, many);
    CUtensorMap qmap, kmap, vmap;
    SLLM_REQUIRE(pt_query_map(&qmap, q, (uint64_t)num_tokens, nq, qs, p.pack_log2, dtype) &&
                 pt_map(&kmap, k_cache, (uint64_t)cache_rows, PT_D, PT_D, PT_PAGE, dtype) &&
                 pt_map(&vmap, v_cache, (uint64_t)cache_rows, PT_D, PT_D, PT_PAGE, dtype),
                 "prefill_attention_paged: cuTensorMapEncodeTiled failed");
    SLLM_DISPATCH_DTYPE(dtype, {
        static unsigned long long configured = 0;
        if (first_use_on_this_device(configured)) {
            cudaFuncSetAttribute(prefill_attn_tc_kernel<T, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM_BYTES);
            cudaFuncSetAttribute(prefill_attn_tc_kernel<T, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM_BYTES);
        }
        if (many) launch_early(prefill_attn_tc_kernel<T, true, true>, grid, PT_THREADS, PT_SMEM_BYTES, stream, qmap, kmap, vmap, p, pg);
        else launch_early(prefill_attn_tc_kernel<T, true, false>, grid, PT_THREADS, PT_SMEM_BYTES, stream, qmap, kmap, vmap, p, pg);
    });
    if (check_launch("prefill_attention_paged(tcgen05)")) return 1;
    if (pg.nsplit > 1) {
        const dim3 rows((unsigned)cdiv((int64_t)max_chunk_len * nq, 8), (unsigned)num_seqs);
        SLLM_DISPATCH_DTYPE(dtype, (launch_early(prefill_merge_kernel<T>, rows, 256, 0, stream, pg.part_o, pg.part_ml, (T*)o, start_locs, chunk_lens, nq, num_tokens * nq, pg.nsplit)));
        return check_launch("prefill_attention_paged(merge)");
    }
    return 0;
}

}  // namespace sllm

using namespace sllm;

static int prefill_attention_paged(const void* q, const void* k_cache, const void* v_cache, void* o,
                                            const int32_t* block_table, const int32_t* seq_ids,
                                            const int32_t* prefill_seq_start_locs, const int32_t* prefill_seq_lens,
                                            const int32_t* prefill_prefix_lens, float softmax_scale, int num_prefill_seqs,
                                            int max_prefill_len, int64_t num_prefill_tokens, int cur_layer, int num_layers,
                                            int nq, int nkv, int block_size, int head_dim, int max_blocks_per_seq,
                                            int64_t num_blocks, int64_t q_row_stride, sllm_dtype_t dtype, sllm_stream_t stream,
                                   int num_splits, void* workspace) {
    SLLM_REQUIRE(num_prefill_seqs >= 0 && max_prefill_len >= 0, "prefill_attention_paged: negative sizes");
    if (num_prefill_seqs == 0 || max_prefill_len == 0) return 0;
    SLLM_REQUIRE(q && k_cache && v_cache && o && block_table && seq_ids && prefill_seq_start_locs && prefill_seq_lens &&
                 prefill_prefix_lens, "prefill_attention_paged: null pointer");
    SLLM_REQUIRE(head_dim == 64 || head_dim == 128, "prefill_attention_paged: head_dim %d not supported (64, 128)", head_dim);
    SLLM_REQUIRE(nkv > 0 && nq % nkv == 0, "prefill_attention_paged: nq %d not a multiple of nkv %d", nq, nkv);
    SLLM_REQUIRE(q_row_stride >= (int64_t)nq * head_dim && q_row_stride % 8 == 0, "prefill_attention_paged: bad q row stride");
    SLLM_REQUIRE(block_size > 0 && num_layers > 0 && cur_layer >= 0 && cur_layer < num_layers && max_blocks_per_seq > 0 && num_blocks > 0,
                 "prefill_attention_paged: bad cache geometry (layer %d of %d)", cur_layer, num_layers);
    cudaStream_t st = (cudaStream_t)stream;
    // SLLM_PREFILL_ATTN_GEN=1 forces the cp.async/mma.sync kernel (A/B measurements), like sllm_prefill_attention
    const char* gen_env = getenv("SLLM_PREFILL_ATTN_GEN");
    const int gen = (gen_env && gen_env[0] == '1') ? 1 : (gen_env && gen_env[0] == '2') ? 2 : 0;
    const int64_t cache_rows = num_blocks * num_layers * nkv * block_size;
    if (gen != 1 && dtype <= SLLM_BF16 && tc_prefill_paged_supported(head_dim, block_size, num_prefill_tokens, cache_rows)) {
        PtPaged pg{block_table, seq_ids, prefill_prefix_lens, cur_layer, num_layers, max_blocks_per_seq, 1, num_prefill_tokens, nullptr, nullptr};
        if (num_splits > 1 && workspace != nullptr && (int64_t)num_prefill_seqs * num_splits <= 65535) {
            pg.nsplit = num_splits; pg.part_o = (float*)workspace; pg.part_ml = pg.part_o + (int64_t)num_splits * num_prefill_tokens * nq * PT_D;
        }
        return launch_prefill_paged_tc(q, k_cache, v_cache, o, prefill_seq_start_locs, prefill_seq_lens,
                                       softmax_scale * 1.4426950408889634f, num_prefill_seqs, max_prefill_len, num_prefill_tokens,
                                       nq, nkv, q_row_stride, cache_rows, pg, dtype, st);
    }
    SLLM_REQUIRE(gen != 2, "prefill_attention_paged: SLLM_PREFILL_ATTN_GEN=2 but the shape is not covered by the tcgen05 kernel");
    PfPagedKV pk{block_table, seq_ids, prefill_prefix_lens, cur_layer, num_layers, block_size, max_blocks_per_seq};
    if (head_dim == 128) { SLLM_DISPATCH_DTYPE(dtype, return (launch_prefill_paged<T, 128>(q, k_cache, v_cache, o, prefill_seq_start_locs, prefill_seq_lens, softmax_scale, num_prefill_seqs, max_prefill_len, nq, nkv, q_row_stride, pk, st))); }
    else { SLLM_DISPATCH_DTYPE(dtype, return (launch_prefill_paged<T, 64>(q, k_cache, v_cache, o, prefill_seq_start_locs, prefill_seq_lens, softmax_scale, num_prefill_seqs, max_prefill_len, nq, nkv, q_row_stride, pk, st))); }
    return 0;
}

extern "C" int sllm_prefill_attention_paged(
    const void* q, const void* k_cache, const void* v_cache, void* o,
    const int32_t* block_table, const int32_t* seq_ids,
    const int32_t* prefill_seq_start_locs, const int32_t* prefill_seq_lens,
    const int32_t* prefill_prefix_lens, float softmax_scale, int num_prefill_seqs,
    int max_prefill_len, int64_t num_prefill_tokens, int cur_layer, int num_layers,
    int nq, int nkv, int block_size, int head_dim, int max_blocks_per_seq,
    int64_t num_blocks, int64_t q_row_stride, sllm_dtype_t dtype, sllm_stream_t stream) {
    return prefill_attention_paged(q, k_cache, v_cache, o, block_table, seq_ids, prefill_seq_start_locs, prefill_seq_lens,
                                   prefill_prefix_lens, softmax_scale, num_prefill_seqs, max_prefill_len, num_prefill_tokens,
                                   cur_layer, num_layers, nq, nkv, block_size, head_dim, max_blocks_per_seq, num_blocks,
                                   q_row_stride, dtype, stream, 1, nullptr);
}

extern "C" int sllm_prefill_attention_paged_split(
    const void* q, const void* k_cache, const void* v_cache, void* o,
    const int32_t* block_table, const int32_t* seq_ids,
    const int32_t* prefill_seq_start_locs, const int32_t* prefill_seq_lens,
    const int32_t* prefill_prefix_lens, float softmax_scale, int num_prefill_seqs,
    int max_prefill_len, int64_t num_prefill_tokens, int cur_layer, int num_layers,
    int nq, int nkv, int block_size, int head_dim, int max_blocks_per_seq,
    int64_t num_blocks, int64_t q_row_stride, sllm_dtype_t dtype, sllm_stream_t stream,
    int num_splits, void* workspace) {
    SLLM_REQUIRE(num_splits >= 1 && num_splits <= 64, "prefill_attention_paged: 1 <= splits <= 64 (got %d)", num_splits);
    return prefill_attention_paged(q, k_cache, v_cache, o, block_table, seq_ids, prefill_seq_start_locs, prefill_seq_lens,
                                   prefill_prefix_lens, softmax_scale, num_prefill_seqs, max_prefill_len, num_prefill_tokens,
                                   cur_layer, num_layers, nq, nkv, block_size, head_dim, max_blocks_per_seq, num_blocks,
                                   q_row_stride, dtype, stream, num_splits, workspace);
}
