// Causal varlen prefill attention, generation 2 (tcgen05 + TMA): host side of the packed-k/v variant.  The kernel is
// prefill_attn_tc_kernel.cuh; reference being replaced: swiftllm/worker/kernels/prefill_attn.py:9-139 and the
// flash_attn_varlen_func call at swiftllm/worker/layers/transformer_layer.py:86-96.
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "prefill_attn_tc_kernel.cuh"

namespace sllm {

// ------------------------------------------------------------------ host side
namespace {
std::mutex g_pt_mutex;
struct PtKey {
    const void* ptr; uint64_t rows; int cols; int dt; int64_t stride;
    bool operator==(const PtKey& o) const { return ptr == o.ptr && rows == o.rows && cols == o.cols && dt == o.dt && stride == o.stride; }
};
struct PtKeyHash { size_t operator()(const PtKey& k) const { return std::hash<const void*>()(k.ptr) ^ (k.rows * 1315423911u) ^ (size_t)(k.cols * 31 + k.dt) ^ ((size_t)k.stride << 7); } };
std::unordered_map<PtKey, CUtensorMap, PtKeyHash> g_pt_maps;
}  // namespace

// `rank` dimensions of 16-bit entries, SWIZZLE_128B (cached per (pointer, geometry))
static bool pt_encode(CUtensorMap* out, const PtKey& key, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
    {
        std::lock_guard<std::mutex> lk(g_pt_mutex);
        auto it = g_pt_maps.find(key);
        if (it != g_pt_maps.end()) { *out = it->second; return true; }
    }
    TensorMapEncodeFn enc = get_tensor_map_encoder();
    if (!enc) return false;
    const cuuint32_t es[3] = {1, 1, 1};
    CUresult r = enc(out, key.dt == SLLM_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(key.ptr),
                     dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return false;
    std::lock_guard<std::mutex> lk(g_pt_mutex);
    if (g_pt_maps.size() > 4096) g_pt_maps.clear();
    g_pt_maps[key] = *out;
    return true;
}

bool pt_map(CUtensorMap* out, const void* ptr, uint64_t rows, int cols, int64_t row_stride, int box_rows, sllm_dtype_t dt) {
    const cuuint64_t dims[2] = {(cuuint64_t)cols, rows}, strides[1] = {(cuuint64_t)row_stride * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    return pt_encode(out, PtKey{ptr, rows, cols * 1024 + box_rows, (int)dt, row_stride}, 2, dims, strides, box);
}

bool pt_query_map(CUtensorMap* out, const void* ptr, uint64_t rows, int heads, int64_t row_stride, int pack_log2, sllm_dtype_t dt) {
    const cuuint64_t dims[3] = {PT_D, (cuuint64_t)heads, rows}, strides[2] = {PT_D * 2, (cuuint64_t)row_stride * 2};
    const cuuint32_t box[3] = {64, 1u << pack_log2, (cuuint32_t)PT_BQ >> pack_log2};
    return pt_encode(out, PtKey{ptr, rows, -(heads * 1024 + pack_log2), (int)dt, row_stride}, 3, dims, strides, box);
}

// Up to eight query heads of a key/value head lie side by side in a tile: rows of fewer tokens, so that a tile of 128 rows multiplies fewer keys that most
// of its rows do not see, and short prompts fill their tiles.
static int pt_pack_log2(int nq, int nkv) {
    int n = 0;
    while (n < 3 && (nq / nkv) % (2 << n) == 0) n++;
    return n;
}
// Query blocks of one or two tiles of all sequences, for one of the heads / pack: every sequence ends in a block of its own
static int64_t pt_blocks_of_all(int pack_log2, int num_seqs, int max_len, int64_t num_tokens, int tiles) {
    const int tokens = tiles * PT_BQ >> pack_log2;
    return std::min<int64_t>((int64_t)num_seqs * cdiv(max_len, tokens), num_tokens / tokens + num_seqs);
}

// Blocks of one tile where that leaves no SM two of them (a step of one tile ends sooner: a prompt of 300 tokens, 32 / 8 heads, 9.0 us, with two tiles 11.3),
// or few of them that are short (20 prompts of up to 200 tokens, 16 / 4 heads: 14.4, with two 16.6; at 64 / 8 heads, seven an SM, 32.9 and 31.9).
dim3 pt_grid(PtParams& p, int num_seqs, int max_len, int64_t num_tokens, int nsplit, bool paged, bool& many) {
    static int sm_count[64];                                   // by device
    const int dev = current_device() & 63;
    int sms = __atomic_load_n(&sm_count[dev], __ATOMIC_RELAXED);
    if (sms == 0) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, current_device());
        __atomic_store_n(&sm_count[dev], sms, __ATOMIC_RELAXED);
    }
    p.pack_log2 = pt_pack_log2(p.nq, p.nkv);
    p.num_seqs = num_seqs; p.order = PT_AT_ONCE;
    const int64_t heads = p.nq >> p.pack_log2;
    const int whole = cdiv(max_len, 2 * PT_BQ) * 2 * PT_BQ;    // rows up to the whole 256 behind the longest that the caller states
    auto blocks = [&](int tiles) { return pt_blocks_of_all(p.pack_log2, num_seqs, max_len, num_tokens, tiles); };
    const int64_t ones = heads * nsplit * blocks(1);
    p.tiles = ones <= sms || (!paged && max_len <= 4 * PT_BK && 2 * ones <= 5 * sms) ? 1 : 2;
    const int tokens = p.tiles * PT_BQ >> p.pack_log2, each = cdiv(max_len, tokens);
    p.max_blocks = whole / tokens;
    // a few short items over: their CTAs end sooner than the grid's next one is asked for (152 of up to four steps: 13.4 us, launched 11).  Portions
    // whose blocks all find an SM: a CTA for each, which need not search, beside a few without a block (us, searched / launched: six of up to
    // 400 tokens at 200, 16 / 4 heads, 17.3 / 16.3; four of up to 300 at 500, 16 / 16 heads, 15.9 / 14.9; two of up to 100 at 4000, 24 / 4 heads, 23.1 / 24.0)
    const bool launched = paged ? heads * nsplit * blocks(p.tiles) <= sms : max_len <= 4 * PT_BK;
    many = heads * num_seqs * nsplit * each > (!launched ? sms : paged ? 3 * sms / 2 : 2 * sms);
    if (!many) return dim3((unsigned)each, (unsigned)heads, (unsigned)(num_seqs * nsplit));
    const unsigned slots = (unsigned)std::min<int64_t>(blocks(p.tiles) * nsplit, 65535);
    // Portions of a few items an SM end on the shortest items of all heads, not on the last head's long ones.  With more, the items of a head together:
    // their keys stay in L2 (us, heads apart / together: 4 portions of up to 1024 tokens at 1000, 16 / 16 heads, 160 items, 43 / 52, 32 / 8 heads, 288
    // items, 56 / 65; 16 of up to 300 at 3000, 24 / 4 heads, 348 items, 134 / 138; 32 of up to 500 at 4000, 32 / 8 heads, 1136 items, 573 / 517)
    p.order = !paged ? PT_BY_HEAD : heads * slots <= sms ? PT_AT_ONCE : heads * slots <= 4 * sms ? PT_BY_HEAD : PT_BY_SLOT;
    return p.order == PT_BY_HEAD ? dim3((unsigned)heads, slots) : dim3(slots, (unsigned)heads);
}

bool tc_prefill_supported(int head_dim, int64_t num_tokens) {
    return head_dim == PT_D && num_tokens > 0 && num_tokens < (1LL << 31) && get_tensor_map_encoder() != nullptr;
}

int launch_prefill_tc(const void* q, const void* k, const void* v, void* o, const int32_t* start_locs, const int32_t* seq_lens,
                      float scale_log2e, int num_seqs, int max_len, int64_t num_tokens, int nq, int nkv, int64_t qs, int64_t ks,
                      int64_t vs, sllm_dtype_t dtype, cudaStream_t stream) {
    PtParams p;
    p.o = o; p.start_locs = start_locs; p.seq_lens = seq_lens; p.scale_log2e = scale_log2e; p.nq = nq; p.nkv = nkv;
    bool many;
    const dim3 grid = pt_grid(p, num_seqs, max_len, num_tokens, 1, false, many);
    CUtensorMap qmap, kmap, vmap;
    SLLM_REQUIRE(pt_query_map(&qmap, q, (uint64_t)num_tokens, nq, qs, p.pack_log2, dtype) &&
                 pt_map(&kmap, k, (uint64_t)num_tokens, nkv * PT_D, ks, PT_BK, dtype) &&
                 pt_map(&vmap, v, (uint64_t)num_tokens, nkv * PT_D, vs, PT_BK, dtype),
                 "prefill_attention: cuTensorMapEncodeTiled failed");
    SLLM_DISPATCH_DTYPE(dtype, {
        static unsigned long long configured = 0;
        if (first_use_on_this_device(configured)) {
            cudaFuncSetAttribute(prefill_attn_tc_kernel<T, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM_BYTES);
            cudaFuncSetAttribute(prefill_attn_tc_kernel<T, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM_BYTES);
        }
        // (begun early or not, us called eagerly: eight prompts of up to 600 tokens, 32 / 8 heads, 28.7 / 31.4, twelve of up to 1777, 16 / 4 heads, 70.0 / 72.1,
        // 4 x 4096, 32 / 8 heads, 477 / 476)
        if (many) launch_early(prefill_attn_tc_kernel<T, false, true>, grid, PT_THREADS, PT_SMEM_BYTES, stream, qmap, kmap, vmap, p, PtPaged{});
        else launch_early(prefill_attn_tc_kernel<T, false, false>, grid, PT_THREADS, PT_SMEM_BYTES, stream, qmap, kmap, vmap, p, PtPaged{});
    });
    return check_launch("prefill_attention(tcgen05)");
}

}  // namespace sllm

extern "C" int64_t sllm_prefill_attention_blocks(int nq, int nkv, int num_prefill_seqs, int max_prefill_len, int64_t num_prefill_tokens, int tiles) {
    using namespace sllm;
    if (nkv <= 0 || nq <= 0 || nq % nkv != 0 || num_prefill_seqs <= 0 || max_prefill_len <= 0 || num_prefill_tokens < 0 || tiles < 1 || tiles > 2) return 0;
    const int pack_log2 = pt_pack_log2(nq, nkv);
    return (nq >> pack_log2) * pt_blocks_of_all(pack_log2, num_prefill_seqs, max_prefill_len, num_prefill_tokens, tiles);
}
