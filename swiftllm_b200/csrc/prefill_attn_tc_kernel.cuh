// Causal varlen prefill attention, tcgen05 + TMA kernel, two query tiles per CTA in ping-pong (sm_100a).
// Shared by prefill_attn_tc.cu (packed k/v of the batch) and prefill_attn_paged.cu (chunked prefill: K/V pages gathered
// from the KV cache through the block table).
//
// Reference being replaced: swiftllm/worker/kernels/prefill_attn.py:9-139 and the flash_attn_varlen_func call at
// swiftllm/worker/layers/transformer_layer.py:86-96.  head_dim 128, fp16/bf16: fp32 scores, exp2 online softmax in fp32, P rounded
// to the storage dtype before P.V, o = h(acc / l).
//
// ITEM = 256 query rows of a sequence = two 128-row tiles A and B, keys in steps of 80; row = (token, head), with the query heads of one
// key/value head side by side (`pack`).  CTAs are persistent: an item's last softmax, its last products and its output run beside the next
// item's loads and first products.  Three warpgroups:
//   warp 0 / 2  TMA producers: warp 0 finds the items, loads Q (4 boxes of 128 rows x 64 d) and then the K tiles, warp 2 the V tiles
//               (2 boxes of 80 x 64 per step) into separate four-stage rings with their own mbarriers, which run on from item to item.
//   warp 1 / 3  product issuers of tile A / B (one elected lane):  S_X(j + 1) = Q_X . K(j + 1) as soon as the softmax warps hold S_X(j)
//               in registers (8 UMMAs, M = 128 N = 80 K = 16), O_X += P_X(j) . V(j) when P_X(j) is there (5 UMMAs, N = 128, B MN-major).
//   warps 4-7   softmax of tile A, warps 8-11 softmax of tile B: thread = query row = TMEM lane.  Row max and row sum
//               are thread-local (no shuffles); P goes back into TMEM as the A operand of P . V.
//               O is rescaled in TMEM only when the running max grew by more than 2^8 ("lazy rescale": the
//               reference point m_ref trails the true max, exact in the end because l uses the same reference).
// TMEM: S_A 0..79, S_B 80..159, P_A 160..199, P_B 200..239, O_A 256..383, O_B 384..511.
//
// Items come from the launch's grid, the longest first: a CTA that is about to finish one takes a CTA that has not been launched yet in its own
// stead (cluster launch control), so that the SMs share the items as they get to them whatever the lengths are, and beside other kernels.  It asks
// when the last PT_STAGES steps' keys are yet to load: asked at an item's beginning, the CTAs of the longest items, which begin first, had taken a
// second one before the others ended (us, at the beginning / now: one prompt of 4096 tokens, 16 / 4 heads, 85 / 64; two of up to 2000, 32 / 8
// heads, 51 / 41; three of up to 1000, 64 / 8 heads, 44 / 45.6; twelve of up to 1777, 16 / 4 heads, 72 both; launched late, as both were then).  Portions in no more CTAs
// than SMs do not ask: a request that finds none costs their steps 7 % (one of 1024 tokens at 5000, 24 / 4 heads, 93 us with and 87 without).
// With a CTA per (sequence, head, 256 tokens) 4000 cycles passed before its first product, over a quarter of a prompt of 450 tokens, and a tile's rows
// multiplied 104 keys on the average that they do not see, now 56 at four heads a tile.  Measured on B200, us: 4 x 4096 bf16, 32 / 8 heads 590 -> 544
// (1010 TFLOP/s), twelve ragged fp16 prompts of up to 1777 tokens 202 -> 157, 64 of up to 100 tokens 72 -> 29, 512 tokens at 3584 47.2 -> 45.3.
// An issuer works out its operands before it waits: it sits between every softmax and the products behind it (3 to 6 %).
//
// Why steps of 80 keys: scores and P need places of their own, so that the next scores are multiplied while the softmax of the last ones
// runs.  With 128 keys P has to lie over its scores (TMEM is full), which chains S, softmax and P . V of a tile one after the other: 3510
// cycles a step where products and exponentials each need 2048.  80 keys are the most that leave room for both.
// Roofline: tensor-bound; FLOPs = 4 * nq * D * sum_i L_i (L_i + 1) / 2.
#pragma once
#include "tc_helpers.cuh"

namespace sllm {

using namespace tc;

constexpr int PT_D = 128;
constexpr int PT_BQ = 128;                // rows per query tile (two tiles per CTA)
constexpr int PT_BK = 80;                 // kv tokens per pipeline step
constexpr int PT_STAGES = 4;              // K and V rings (separate producers)
constexpr int PT_THREADS = 384;           // warp 0 Q + K producer, 1 products, 2 V producer, 4-7 softmax A, 8-11 softmax B
constexpr int PT_Q_BYTES = PT_BQ * PT_D * 2;          // 32 KiB per query tile ([half][128 rows][128 B])
constexpr int PT_KV_BYTES = PT_BK * PT_D * 2;         // 20 KiB per K (or V) tile ([half][80 rows][128 B])
constexpr int PT_SMEM_BYTES = 2 * PT_Q_BYTES + 2 * PT_STAGES * PT_KV_BYTES + 1024;
constexpr int PT_TMEM_COLS = 512;
constexpr int PT_S_COL = 0, PT_P_COL = 160, PT_O_COL = 256;      // tile B: + 80, + 40, + 128
constexpr float PT_RESCALE_THRESHOLD = 8.0f;          // log2 units
// registers: 384 threads are launched with 168 each; the softmax warpgroups hold a row of scores and of P
constexpr int PT_REGS_FEW = 88, PT_REGS_MANY = 208;
static_assert(PT_REGS_FEW + 2 * PT_REGS_MANY <= 3 * 168, "the warpgroups' shares must fit what the block was launched with");

constexpr int PT_CONSUMERS = 11;          // warps that read an item: issuers, V producer, softmax

struct PtBarriers {
    uint64_t q_full, q_empty, next;
    uint64_t item_full[2], item_empty[2];                       // [slot]
    uint64_t k_full[PT_STAGES], k_empty[PT_STAGES], v_full[PT_STAGES], v_empty[PT_STAGES];
    uint64_t s_full[2], s_empty[2], p_full[2], p_empty[2], o_empty[2];      // [tile]
};

enum PtOrder { PT_AT_ONCE, PT_BY_SLOT, PT_BY_HEAD };      // portions whose CTAs all have an SM; others: grid (slots, heads) or (heads, slots)

struct PtParams {
    void* o;
    const int32_t* start_locs; const int32_t* seq_lens;
    float scale_log2e;
    int nq, nkv;
    int pack_log2;                        // query heads of one key/value head that lie side by side in a tile
    int num_seqs, tiles, max_blocks;      // query blocks of one or two tiles; those of a sequence that count
    int order;                            // of a MANY launch: a PtOrder
};
// what the warps of a CTA have to know of an item; tile A takes part in nkt_a steps of 80 keys, B in nkt_b, from step j0 on
struct PtItem {
    int valid, tok0, len, q0, head0, seq_id, pre, split, j0, nkt_a, nkt_b;
    __device__ __forceinline__ int steps() const { return max(nkt_a, nkt_b); }
    __device__ __forceinline__ int steps_of(int tile) const { return tile == 0 ? nkt_a : nkt_b; }
};

// PAGED launches (chunked prefill): where the keys / values live.  kmap / vmap then describe the paged caches as
// [num_blocks * L * nkv * 16 rows, 128] with boxes of (64 d x 16 tokens) = one d-half of one page.
struct PtPaged {
    const int32_t* block_table; const int32_t* seq_ids; const int32_t* prefix_lens;
    int cur_layer, num_layers, max_blocks_per_seq;
    // key splits (steps with few query blocks): slot = query block * nsplit + split, without MANY blockIdx.z = sequence * nsplit + split; nsplit > 1
    // leaves fp32 rows of unnormalised O [nsplit, tokens, nq, 128] and their (reference maximum in base 2, sum) [nsplit, tokens, nq, 2] for prefill_merge_kernel
    int nsplit; int64_t num_tokens;
    float* part_o; float* part_ml;
};
constexpr int PT_PAGE = 16;               // tokens per KV page (PAGED only)

// All sequences' query blocks, those of the highest rows first (they have the most keys).  Each by a whole warp
__device__ __forceinline__ int pt_blocks(const PtParams& p, int s, int len) {            // of sequence s, which has that many rows
    const int log2 = (p.tiles == 2 ? 8 : 7) - p.pack_log2;
    return s < p.num_seqs ? min((max(len, 0) + (1 << log2) - 1) >> log2, p.max_blocks) : 0;
}
static_assert(PT_BQ == 128, "rows of a block");
__device__ __forceinline__ int pt_blocks_from(const PtParams& p, int mine, int b) {      // blocks b and up of every sequence; mine: the lane's sequence
    int n = max(mine - b, 0);
    for (int s = 32 + (threadIdx.x & 31); s < p.num_seqs; s += 32) n += max(pt_blocks(p, s, p.seq_lens[s]) - b, 0);
    return (int)__reduce_add_sync(0xffffffffu, (unsigned)n);
}
// A CTA's ranks grow, but for a step back where its next head's begin: the search goes on where the last one ended, among the sequences that have a
// block of the same number, and halves the numbers only outside of them.  (Started afresh for every item it read all lengths several times an item.  us,
// afresh / now: 1000 prompts of up to 60 tokens, 16 / 16 heads 561 / 280; 2000 of up to 30 1703 / 538; 256 of up to 100, 32 / 8 heads 110 / 96; up to
// 32 sequences, whose counts the lanes hold, are not affected.)
struct PtCursor { int block, first, count, s0, before; };      // the sequences that have `block`: ranks first .. + count - 1, `before` of them in front of sequence s0
__device__ __forceinline__ int pt_block(const PtParams& p, int mine, int total, int rank, PtCursor& c) {      // the sequence of that rank's block; rank < total
    const int lane = threadIdx.x & 31;
    if (rank < c.first || rank >= c.first + c.count) {
        int lo = 0, hi = p.max_blocks, from_lo = total, from_hi = 0;      // blocks from lo on are more than `rank`, from hi on not
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1, n = pt_blocks_from(p, mine, mid);
            if (n > rank) { lo = mid; from_lo = n; }
            else { hi = mid; from_hi = n; }
        }
        c = PtCursor{lo, from_hi, from_lo - from_hi, 0, 0};
    } else if (rank < c.first + c.before) c.s0 = c.before = 0;
    const int r = rank - c.first;                                     // the r-th of those that have it
    for (; c.s0 < p.num_seqs; c.s0 += 128) {
        bool has[4];                                                  // (four loads in flight)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int s = c.s0 + 32 * k + lane;
            has[k] = (s < 32 ? mine : pt_blocks(p, s, s < p.num_seqs ? p.seq_lens[s] : 0)) > c.block;
        }
        int n = c.before;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t all = __ballot_sync(0xffffffffu, has[k]);
            const uint32_t it = __ballot_sync(0xffffffffu, has[k] && n + __popc(all & ((1u << lane) - 1u)) == r);
            if (it) return c.s0 + 32 * k + __ffs(it) - 1;
            n += __popc(all);
        }
        c.before = n;
    }
    return 0;                                                         // (not reached: a rank below the total has its sequence)
}

// PAGED = false: K/V tiles come from the packed k/v rows of the batch (the reference's contract).
// PAGED = true (chunked prefill): the chunk's queries sit at positions prefix .. prefix + len - 1 of
// their sequence; every 80-token K/V step is gathered from five 16-token pages of the KV cache through the block
// table (lanes 0-4 of the producer warp issue the two d-half boxes of one page each), landing in the SAME
// [half][80 rows][128 B] layout, so the product issuer and its descriptors are shared by both variants.  Page slots that a tail step does not
// load keep what lay there: their scores are masked, and P . V stops before them.
// MANY: more items than SMs.  grid: heads / pack and slots (all sequences' query blocks; a CTA takes every so many, if they are more than the grid
// has).  The order of the grid is the order of the work: (heads, slots), the longest items of all heads first, for packed prompts and for portions
// of up to four items an SM; (slots, heads) for other portions, whose keys may be more than L2 holds.  Else grid (query blocks from the last
// one, heads / pack, sequence * nsplit + split), a CTA for an item.
template <typename T, bool PAGED, bool MANY>
__global__ void __launch_bounds__(PT_THREADS, 1) prefill_attn_tc_kernel(const __grid_constant__ CUtensorMap qmap,
                                                                        const __grid_constant__ CUtensorMap kmap,
                                                                        const __grid_constant__ CUtensorMap vmap,
                                                                        const PtParams p, const PtPaged pg) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* q_sm = smem;                                       // [2 tiles][2 halves][128 rows][128 B]
    uint8_t* k_sm = q_sm + 2 * PT_Q_BYTES;                      // [stage][2 halves][80 rows][128 B]
    uint8_t* v_sm = k_sm + PT_STAGES * PT_KV_BYTES;
    uint8_t* misc = v_sm + PT_STAGES * PT_KV_BYTES;
    PtBarriers* bars = reinterpret_cast<PtBarriers*>(misc);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(misc + 512);
    PtItem* items = reinterpret_cast<PtItem*>(misc + 528);      // two slots
    uint8_t* answer = misc + 640;
    static_assert(sizeof(PtBarriers) <= 512 && 528 + 2 * sizeof(PtItem) <= 640, "barriers, items and the answer share a kilobyte");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    wait_previous();
    if (!PAGED || pg.nsplit == 1) launch_next();                // (a merge begins as the CTAs end: it would gather on the idle SMs; 64 tokens at 3000: 18.6 -> 17.2 us)
    const int nsplit = PAGED ? pg.nsplit : 1;
    const int tile_tokens = PT_BQ >> p.pack_log2;

    // what warp 0 knows: the slot, how many there are, the lane's sequence (without MANY: the CTA's)
    const bool takes = MANY && (!PAGED || p.order != PT_AT_ONCE), by_head = MANY && (!PAGED || p.order == PT_BY_HEAD);
    int head_block = by_head ? blockIdx.x : blockIdx.y, slot = by_head ? blockIdx.y : MANY ? blockIdx.x : gridDim.x - 1 - blockIdx.x, slots = 0;
    const int slot_step = by_head ? gridDim.y : gridDim.x;
    PtCursor cursor = {0, 0, 0, 0, 0};
    int mine = lane, my_split = 0, my_blocks = 0, my_len = 0, my_start = 0, my_pre = 0, my_id = 0;
    if constexpr (!MANY) {
        mine = blockIdx.z;
        if (PAGED && nsplit > 1) { mine = blockIdx.z / nsplit; my_split = blockIdx.z - mine * nsplit; }
    }
    auto find = [&]() {                                         // the item of `slot` of all `slots`
        PtItem it;
        it.valid = slot < slots;
        it.len = my_len; it.tok0 = my_start; it.pre = my_pre; it.seq_id = my_id; it.split = my_split;
        int block = slot;
        if constexpr (MANY) {
            if (!it.valid) return it;
            const int seq = pt_block(p, my_blocks, slots / nsplit, PAGED ? slot / nsplit : slot, cursor);
            block = cursor.block;
            it.split = PAGED ? slot % nsplit : 0;
            it.len = __shfl_sync(0xffffffffu, my_len, seq & 31);                         // query rows of this sequence in the batch
            it.tok0 = __shfl_sync(0xffffffffu, my_start, seq & 31);
            it.pre = __shfl_sync(0xffffffffu, my_pre, seq & 31);                         // position of query row 0 within its sequence
            it.seq_id = __shfl_sync(0xffffffffu, my_id, seq & 31);
            if (seq >= 32) {
                it.len = p.seq_lens[seq]; it.tok0 = p.start_locs[seq];
                if constexpr (PAGED) { it.pre = pg.prefix_lens[seq]; it.seq_id = pg.seq_ids[seq]; }
            }
        }
        it.q0 = block * p.tiles * tile_tokens; it.head0 = head_block << p.pack_log2;
        auto upto = [&](int q) { return (it.pre + min(it.len, q) + PT_BK - 1) / PT_BK; };      // kv steps a tile takes part in: up to its last row's key
        const int all_a = upto(it.q0 + tile_tokens), all_b = p.tiles == 2 && it.q0 + tile_tokens < it.len ? upto(it.q0 + 2 * tile_tokens) : 0;
        // the split's steps of them: j0 .. (all of them without splits); the loops below count from j0
        const int per = !PAGED ? 0 : nsplit == 1 ? max(all_a, all_b) : (max(all_a, all_b) + nsplit - 1) / nsplit;
        it.j0 = it.split * per;
        it.nkt_a = PAGED ? min(max(all_a - it.j0, 0), per) : all_a;
        it.nkt_b = PAGED ? min(max(all_b - it.j0, 0), per) : all_b;
        return it;
    };
    auto load_queries = [&](const PtItem& it) {
        const uint32_t qbar = smem_u32(&bars->q_full);
        mbar_arrive_expect_tx(qbar, p.tiles * PT_Q_BYTES);
        for (int x = 0; x < p.tiles; x++)
            for (int h = 0; h < 2; h++)
                tma_load_3d(smem_u32(q_sm + x * PT_Q_BYTES + h * (PT_Q_BYTES / 2)), &qmap, qbar, h * 64, it.head0, it.tok0 + it.q0 + x * tile_tokens);
    };

    PtItem first;
    if (warp == 2 && lane == 0) { tma_prefetch_desc(&qmap); tma_prefetch_desc(&kmap); tma_prefetch_desc(&vmap); }
    if (warp == 0) {
        if (mine < p.num_seqs) {
            my_len = p.seq_lens[mine]; my_start = p.start_locs[mine];
            if constexpr (PAGED) { my_pre = pg.prefix_lens[mine]; my_id = pg.seq_ids[mine]; }
        }
        if (lane == 0) {
            mbar_init(smem_u32(&bars->q_full), 1); mbar_init(smem_u32(&bars->q_empty), 2); mbar_init(smem_u32(&bars->next), 1);
            for (int i = 0; i < 2; i++) { mbar_init(smem_u32(&bars->item_full[i]), 1); mbar_init(smem_u32(&bars->item_empty[i]), PT_CONSUMERS); }
            for (int i = 0; i < PT_STAGES; i++) {
                mbar_init(smem_u32(&bars->k_full[i]), 1); mbar_init(smem_u32(&bars->k_empty[i]), 2);
                mbar_init(smem_u32(&bars->v_full[i]), 1); mbar_init(smem_u32(&bars->v_empty[i]), 2);
            }
            for (int x = 0; x < 2; x++) {
                mbar_init(smem_u32(&bars->s_full[x]), 1); mbar_init(smem_u32(&bars->s_empty[x]), 128);
                mbar_init(smem_u32(&bars->p_full[x]), 128); mbar_init(smem_u32(&bars->p_empty[x]), 1);
                mbar_init(smem_u32(&bars->o_empty[x]), 128);
            }
            mbar_fence_init();
        }
        my_blocks = slots = pt_blocks(p, mine, my_len);
        if constexpr (MANY) slots = pt_blocks_from(p, my_blocks, 0) * nsplit;
        first = find();
        if (lane == 0 && first.valid) load_queries(first);      // (the thread that made the barriers)
        __syncwarp();
    }
    if (warp == 1) tmem_alloc<PT_TMEM_COLS>(smem_u32(tmem_base_s));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_base_s;

    // item n of this CTA, as warp 0 has left it
    auto take = [&](int n) {
        mbar_wait(smem_u32(&bars->item_full[n & 1]), (n >> 1) & 1);
        const PtItem it = items[n & 1];
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars->item_empty[n & 1]));
        return it;
    };

    if (warp < 4) {
        reg_dec<PT_REGS_FEW>();
        const uint32_t next_bar = smem_u32(&bars->next), next_at = smem_u32(answer);
        // An item's steps of a ring; k0: the ring's steps before it; ask_at: the step at which the grid's next CTA is asked for.  PAGED (one whole
        // warp per ring): step j = pages 5j .. 5j+4 of the sequence.  The block-table entries of the NEXT step are fetched before this step's stage
        // is waited for; lane 0 arms the mbarrier with the bytes of the pages that exist, then lanes 0..4 issue the two (64 d x 16 token) boxes of
        // one page each.
        auto paged_producer = [&](const PtItem& it, int k0, const CUtensorMap& map, uint8_t* ring, uint64_t* full, uint64_t* empty, int ask_at) {
            const int32_t* bt = pg.block_table + (int64_t)it.seq_id * pg.max_blocks_per_seq;
            const int kvlen = it.pre + it.len, npages = (kvlen + PT_PAGE - 1) / PT_PAGE, nkt = it.steps();
            const int kvh = it.head0 / (p.nq / p.nkv);
            constexpr int PPS = PT_BK / PT_PAGE;                  // pages per step
            int nxt = (lane < PPS && it.j0 * PPS + lane < npages) ? bt[it.j0 * PPS + lane] : 0;
            for (int j = 0; j < nkt; j++) {
                const int st = (k0 + j) % PT_STAGES;
                const int blk = nxt;
                const int npg = (it.j0 + j + 1) * PPS + lane;
                nxt = (j + 1 < nkt && lane < PPS && npg < npages) ? bt[npg] : 0;
                const int valid = min(PPS, npages - (it.j0 + j) * PPS);      // >= 1: step j exists because page 5j does
                const uint32_t bar = smem_u32(&full[st]);
                if (lane == 0) {
                    if (MANY && j == ask_at) ask_next_cta(next_at, next_bar);
                    mbar_wait(smem_u32(&empty[st]), (((k0 + j) / PT_STAGES) & 1) ^ 1);
                    mbar_arrive_expect_tx(bar, (uint32_t)valid * PT_PAGE * PT_D * 2);
                }
                __syncwarp();
                if (lane < valid) {
                    // row of the cache viewed as [num_blocks * L * nkv * 16 rows, 128]: first token row of this page
                    const int64_t row = (((int64_t)blk * pg.num_layers + pg.cur_layer) * p.nkv + kvh) * PT_PAGE;
                    const uint32_t dst = smem_u32(ring + st * PT_KV_BYTES) + lane * (PT_PAGE * 128);
                    tma_load_2d(dst, &map, bar, 0, (int)row);
                    tma_load_2d(dst + PT_KV_BYTES / 2, &map, bar, 64, (int)row);
                }
            }
        };
        auto packed_producer = [&](const PtItem& it, int k0, const CUtensorMap& map, uint8_t* ring, uint64_t* full, uint64_t* empty, int ask_at) {
            const int nkt = it.steps(), kvh = it.head0 / (p.nq / p.nkv);
            for (int j = 0; lane == 0 && j < nkt; j++) {
                const int st = (k0 + j) % PT_STAGES;
                if (MANY && j == ask_at) ask_next_cta(next_at, next_bar);
                mbar_wait(smem_u32(&empty[st]), (((k0 + j) / PT_STAGES) & 1) ^ 1);
                const uint32_t bar = smem_u32(&full[st]), dst = smem_u32(ring + st * PT_KV_BYTES);
                mbar_arrive_expect_tx(bar, PT_KV_BYTES);
                tma_load_2d(dst, &map, bar, kvh * PT_D, it.tok0 + j * PT_BK);
                tma_load_2d(dst + PT_KV_BYTES / 2, &map, bar, kvh * PT_D + 64, it.tok0 + j * PT_BK);
            }
            __syncwarp();
        };
        if (warp == 0) {
            // ======================================================= items; TMA producer: Q of an item, then its K tiles
            for (int n = 0, k0 = 0, answers = 0;; n++) {
                const PtItem it = n == 0 ? first : find();
                if (lane == 0) {
                    mbar_wait(smem_u32(&bars->item_empty[n & 1]), ((n >> 1) & 1) ^ 1);
                    items[n & 1] = it;
                    mbar_arrive(smem_u32(&bars->item_full[n & 1]));
                }
                __syncwarp();
                if (!it.valid) break;
                if (lane == 0 && n > 0) {
                    mbar_wait(smem_u32(&bars->q_empty), (n & 1) ^ 1);
                    load_queries(it);
                }
                __syncwarp();
                const int ask_at = takes && slot + slot_step >= slots ? max(it.steps() - PT_STAGES, 0) : -1;      // (behind the CTA's last slot alone)
                if constexpr (PAGED) paged_producer(it, k0, kmap, k_sm, bars->k_full, bars->k_empty, ask_at);
                else packed_producer(it, k0, kmap, k_sm, bars->k_full, bars->k_empty, ask_at);
                k0 += it.steps();
                slot += slot_step;
                if (slot < slots) continue;                      // (more query blocks than the grid has: only where sequences share rows)
                slot = slots;
                if (takes) {
                    if (lane == 0 && it.steps() == 0) ask_next_cta(next_at, next_bar);
                    mbar_wait(next_bar, answers++ & 1);
                    int x, y;
                    if (next_cta(next_at, x, y)) { head_block = by_head ? x : y; slot = by_head ? y : x; }
                }
            }
        } else if (warp == 2) {
            // ======================================================= TMA producer: the V tiles (independent of K's progress)
            for (int n = 0, k0 = 0;; n++) {
                const PtItem it = take(n);
                if (!it.valid) break;
                if constexpr (PAGED) paged_producer(it, k0, vmap, v_sm, bars->v_full, bars->v_empty, -1);
                else packed_producer(it, k0, vmap, v_sm, bars->v_full, bars->v_empty, -1);
                k0 += it.steps();
            }
        } else {
            // ======================================================= product issuers: warp 1 for tile A, warp 3 for tile B, so that neither
            // waits for the other tile; the warp stays converged, one elected lane issues
            const int x = warp >> 1;
            constexpr uint32_t IDESC_S = make_instr_desc(128, PT_BK, UmmaFmt<T>::value, 0, 0);
            constexpr uint32_t IDESC_O = make_instr_desc(128, PT_D, UmmaFmt<T>::value, 0, 1);      // B = V, MN-major
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint32_t s_addr = tm + PT_S_COL + x * PT_BK, p_addr = tm + PT_P_COL + x * (PT_BK / 2), o_addr = tm + PT_O_COL + x * 128;
            // Descriptor bases are loop invariants; per UMMA only the 14-bit address field (16-byte units, low word)
            // advances by a compile-time constant (all tiles live below 256 KiB, so no carry into the LBO field).
            const uint64_t dq0 = make_smem_desc(smem_u32(q_sm + x * PT_Q_BYTES), 16, 1024);
            const uint64_t dk0 = make_smem_desc(smem_u32(k_sm), 16, 1024);
            const uint64_t dv0 = make_smem_desc(smem_u32(v_sm), PT_KV_BYTES / 2, 1024);             // MN-major: LBO = d-half stride
            for (int n = 0, k0 = 0, x0 = 0, outputs = 0;; n++) {      // k0, x0: the rings' and the tile's steps of the items before
                const PtItem it = take(n);
                if (!it.valid) break;
                const int nkx = it.steps_of(x), nkt = it.steps();
                const int end = min(it.pre + it.len, it.pre + it.q0 + (x + 1) * tile_tokens) - it.j0 * PT_BK;      // keys the tile can see
                auto scores = [&](int j) {             // S_X(j), once the softmax warps have read the one before
                    const int st = (k0 + j) % PT_STAGES;
                    const uint64_t kd = dk0 + (uint64_t)((st * PT_KV_BYTES) >> 4);
                    mbar_wait(smem_u32(&bars->k_full[st]), ((k0 + j) / PT_STAGES) & 1);
                    if (x0 + j > 0) mbar_wait(smem_u32(&bars->s_empty[x]), (x0 + j - 1) & 1);
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < 8; ks++)    // 16 d per UMMA; d-half = ks / 4
                            umma_ss(s_addr, dq0 + (uint64_t)(((ks >> 2) * (PT_Q_BYTES / 2) + (ks & 3) * 32) >> 4),
                                    kd + (uint64_t)(((ks >> 2) * (PT_KV_BYTES / 2) + (ks & 3) * 32) >> 4), IDESC_S, ks > 0);
                        umma_commit(smem_u32(&bars->s_full[x]));
                        umma_commit(smem_u32(&bars->k_empty[st]));
                        if (j + 1 == nkx) umma_commit(smem_u32(&bars->q_empty));
                    }
                    __syncwarp();
                };
                mbar_wait(smem_u32(&bars->q_full), n & 1);
                if (nkx > 0) scores(0);
                else if (lane == 0) mbar_arrive(smem_u32(&bars->q_empty));
                for (int j = 0; j < nkx; j++) {
                    if (j + 1 < nkx) scores(j + 1);
                    // O_X += P_X(j) V(j): 16 tokens per UMMA, none past the last key the tile can see
                    const int st = (k0 + j) % PT_STAGES, steps = min(PT_BK / 16, (end - j * PT_BK + 15) / 16);
                    const uint64_t vd = dv0 + (uint64_t)((st * PT_KV_BYTES) >> 4);
                    mbar_wait(smem_u32(&bars->v_full[st]), ((k0 + j) / PT_STAGES) & 1);
                    if (j == 0 && outputs++ > 0) mbar_wait(smem_u32(&bars->o_empty[x]), outputs & 1);      // the last O has been read
                    mbar_wait(smem_u32(&bars->p_full[x]), (x0 + j) & 1);
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < PT_BK / 16; k++)
                            if (k < steps) umma_ts(o_addr, p_addr + 8 * k, vd + (uint64_t)((k * 2048) >> 4), IDESC_O, (j > 0 || k > 0) ? 1u : 0u);
                        umma_commit(smem_u32(&bars->v_empty[st]));
                        umma_commit(smem_u32(&bars->p_empty[x]));
                    }
                    __syncwarp();
                }
                // steps that only the other tile takes: hand the stages on once they have been filled (never a phase ahead)
                for (int j = nkx; j < nkt; j++) {
                    const int st = (k0 + j) % PT_STAGES;
                    mbar_wait(smem_u32(&bars->k_full[st]), ((k0 + j) / PT_STAGES) & 1);
                    if (lane == 0) mbar_arrive(smem_u32(&bars->k_empty[st]));
                    mbar_wait(smem_u32(&bars->v_full[st]), ((k0 + j) / PT_STAGES) & 1);
                    if (lane == 0) mbar_arrive(smem_u32(&bars->v_empty[st]));
                }
                k0 += nkt;
                x0 += nkx;
            }
        }
    } else {
        // =========================================================== softmax warps: tile x = 0 (A) / 1 (B)
        reg_inc<PT_REGS_MANY>();
        const int x = (warp - 4) >> 2;
        const int quad = warp & 3;
        const int row = quad * 32 + lane;                 // row within the tile = TMEM lane
        const uint32_t tlane = (uint32_t)(quad * 32) << 16;
        const uint32_t s_addr = tmem + tlane + PT_S_COL + x * PT_BK;
        const uint32_t p_addr = tmem + tlane + PT_P_COL + x * (PT_BK / 2);
        const uint32_t o_addr = tmem + tlane + PT_O_COL + x * 128;
        const float c = p.scale_log2e;
        for (int n = 0, x0 = 0;; n++) {                   // x0: the tile's steps of the items before
            const PtItem it = take(n);
            if (!it.valid) break;
            const int nk_mine = it.steps_of(x), first = it.q0 + x * tile_tokens, kvlen = it.pre + it.len;
            const int qi = first + (row >> p.pack_log2);  // token within the sequence
            const int head = it.head0 + (row & ((1 << p.pack_log2) - 1));
            const int64_t at = (int64_t)(it.tok0 + qi) * p.nq + head;
            float m_ref = -INFINITY, l = 0.f;
            for (int j = 0; j < nk_mine; j++) {
                const int s = x0 + j;
                mbar_wait(smem_u32(&bars->s_full[x]), s & 1);
                tc_fence_after();
                uint32_t r[PT_BK];
                tmem_ld32(s_addr, reinterpret_cast<uint32_t(&)[32]>(r[0]));
                tmem_ld32(s_addr + 32, reinterpret_cast<uint32_t(&)[32]>(r[32]));
                tmem_ld<16>(s_addr + 64, reinterpret_cast<uint32_t(&)[16]>(r[64]));
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->s_empty[x]));

                const int c0 = (it.j0 + j) * PT_BK;
                if (c0 + PT_BK - 1 > it.pre + first || c0 + PT_BK > kvlen) {
                    // column c0+i is visible iff c0+i <= pre+qi and c0+i < kvlen  <=>  i <= lim   (branch-free selects)
                    const int lim = min(it.pre + qi, kvlen - 1) - c0;
#pragma unroll
                    for (int i = 0; i < PT_BK; i++) r[i] = i <= lim ? r[i] : 0xff800000u;        // -inf
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};        // independent chains
#pragma unroll
                for (int i = 0; i < PT_BK; i += 8)
#pragma unroll
                    for (int g = 0; g < 4; g++) mx[g] = max3(mx[g], __uint_as_float(r[i + 2 * g]), __uint_as_float(r[i + 2 * g + 1]));
                // max of the RAW scores (scale > 0 commutes with max)
                const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c);
                // Lazy rescale.  The decision is per row, but tcgen05.ld/st are warp-collective (.sync.aligned): vote, and
                // let rows that do not need it take part with alpha = 1.
                const bool need = m_new > m_ref + PT_RESCALE_THRESHOLD;   // always true on the first tile (m_ref = -inf)
                if (j > 0 && __any_sync(0xffffffffu, need)) {
                    mbar_wait(smem_u32(&bars->p_empty[x]), (s - 1) & 1);       // P . V(j - 1) is done: O is stable
                    tc_fence_after();
                    const float alpha = need ? fast_exp2_tc(m_ref - m_new) : 1.0f;
                    l *= alpha;
#pragma unroll 1
                    for (int cc = 0; cc < 8; cc++) {
                        uint32_t t[16];
                        tmem_ld<16>(o_addr + cc * 16, t);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++) t[i] = __float_as_uint(__uint_as_float(t[i]) * alpha);
                        tmem_st16(o_addr + cc * 16, t);
                    }
                }
                if (need) m_ref = m_new;
                // p = exp2(s*c - m_ref) (<= 2^8), row sum in fp32, P row into TMEM (two keys per column)
                float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                const float sub = PAGED && m_ref == -INFINITY ? 0.f : -m_ref;      // (a split whose keys so far are all behind the row)
                const float2 neg_m = make_float2(sub, sub), c2 = make_float2(c, c);
                uint32_t w[PT_BK / 2];
#pragma unroll
                for (int i = 0; i < PT_BK / 2; i++) {
                    const float2 e = fma2(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), c2, neg_m);
                    const float2 v = make_float2(fast_exp2_tc(e.x), fast_exp2_tc(e.y));
                    ls[i & 1] = add2(ls[i & 1], v);
                    typename Traits<T>::T2 v2 = Traits<T>::from_f2(v);
                    w[i] = *reinterpret_cast<uint32_t*>(&v2);
                }
                if (j > 0) { mbar_wait(smem_u32(&bars->p_empty[x]), (s - 1) & 1); tc_fence_after(); }      // P(j - 1) has been read
                tmem_st32(p_addr, reinterpret_cast<uint32_t(&)[32]>(w[0]));
                tmem_st8(p_addr + 32, reinterpret_cast<uint32_t(&)[8]>(w[32]));
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->p_full[x]));
                l += (ls[0].x + ls[0].y) + (ls[1].x + ls[1].y);
            }
            x0 += nk_mine;
            if (nk_mine > 0) { mbar_wait(smem_u32(&bars->p_empty[x]), (x0 - 1) & 1); tc_fence_after(); }      // the last P . V
            if (PAGED && nsplit > 1) {
                // ---- a split's part of the row
                const int64_t mine = (int64_t)it.split * pg.num_tokens * p.nq + at;
                if (qi < it.len) *reinterpret_cast<float2*>(pg.part_ml + 2 * mine) = make_float2(m_ref, l);
#pragma unroll 1
                for (int cc = 0; cc < 4 && nk_mine > 0; cc++) {
                    uint32_t t[32];
                    tmem_ld32(o_addr + cc * 32, t);
                    tmem_ld_wait();
                    if (qi < it.len) {
#pragma unroll
                        for (int v = 0; v < 32; v += 4)
                            *reinterpret_cast<uint4*>(pg.part_o + mine * PT_D + cc * 32 + v) = make_uint4(t[v], t[v + 1], t[v + 2], t[v + 3]);
                    }
                    __syncwarp();
                }
            } else if (nk_mine > 0) {
                // ---- output: O / l -> global (row qi of this head), only rows inside the sequence
                const float inv = 1.0f / l;
                T* orow = reinterpret_cast<T*>(p.o) + at * PT_D;
#pragma unroll
                for (int cc = 0; cc < 4; cc++) {
                    uint32_t t[32];
                    tmem_ld32(o_addr + cc * 32, t);
                    tmem_ld_wait();
                    if (qi < it.len) {
#pragma unroll
                        for (int v = 0; v < 4; v++) {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                typename Traits<T>::T2 v2 = Traits<T>::from_f2(make_float2(__uint_as_float(t[v * 8 + e * 2]) * inv,
                                                                                            __uint_as_float(t[v * 8 + e * 2 + 1]) * inv));
                                w[e] = *reinterpret_cast<uint32_t*>(&v2);
                            }
                            *reinterpret_cast<uint4*>(orow + cc * 32 + v * 8) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                    __syncwarp();
                }
            }
            tc_fence_before();
            if (nk_mine > 0) mbar_arrive(smem_u32(&bars->o_empty[x]));      // O has been read (an item without steps has none: no phase ahead)
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc<PT_TMEM_COLS>(tmem);
}

// host (prefill_attn_tc.cu): the launch's head packing, blocks and grid; a cached cuTensorMapEncodeTiled of a [rows, cols] 16-bit tensor, boxes of
// (64 cols x box_rows), and of a [rows, heads, 128] one, boxes of (64 d x 2^pack_log2 heads x as many rows as give 128)
dim3 pt_grid(PtParams& p, int num_seqs, int max_len, int64_t num_tokens, int nsplit, bool paged, bool& many);
bool pt_map(CUtensorMap* out, const void* ptr, uint64_t rows, int cols, int64_t row_stride, int box_rows, sllm_dtype_t dt);
bool pt_query_map(CUtensorMap* out, const void* ptr, uint64_t rows, int heads, int64_t row_stride, int pack_log2, sllm_dtype_t dt);

}  // namespace sllm
