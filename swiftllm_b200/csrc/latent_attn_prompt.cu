// Latent attention of prompt rows in 16-bit storage, rows of 512 latent and 64 rotated entries, cache blocks in multiples of 16 tokens: the same
// function as latent_attn.cu and the same split into passes as latent_attn_tc.cu, whose head comments give the definition, the rows and the
// treatment of values that are not finite.
//
// A CTA owns 64 query ROWS, row = (token, head); per tile of 64 keys
//   S[64, 64]    = Q K^T           36 UMMAs, M = 64, N = 64: Q from TMEM, K in shared memory (K-major)
//   O_q[64, 128] = P K[:, 128 q..] q = 0 .. 3, 4 UMMAs each, M = 64, N = 128: P from TMEM, the same key tile (MN-major)
// Every O_q is a tile's own, made from zero; accumulator warps add it to fp32 registers, O = O 2^(m_old - m_new) + O_q.  Rescales therefore cost
// the tensor core nothing: with O in TMEM they stood between one tile's products and the next's, for the reference is the running maximum itself.
//   warp 0        TMA producer: a tile is four boxes of 16 cache rows, (64 d | 8 rows | 9 chunks | row groups of 8), into a ring of three stages
//   warps 1, 2    product issuers, of S and of O_0 .. O_3: one thread's instructions per product take as long as the product (both by one
//                 warp 551 us, by two 512, with a CTA per 64 rows)
//   warps 4-7     softmax: rows 16 w + lane / 4 (a) and + 8 (b), four lanes a row
//   warps 8-15    accumulators, 16 rows of a quadrant each: warps 8-11 O_0 and O_2, 12-15 O_1 and O_3; 128 registers a thread
// TMEM: an M = 64 operand fills 16 of every 32 lanes.  Lanes 0 .. 15: Q in columns 0 .. 287, two buffers of S behind it.  Lanes 16 .. 31: three buffers
// of O_q, two of P.  Q in TMEM frees its 72 KiB for the third stage, and S's products read 2 KiB of shared memory per 32 cycles instead of 4.
//
// Keys in front of the first that the segment sees and behind the last lie in the boxes of the first and the last tile: the producer zeroes their rows.
//
// ITEM = a run of a CTA's tokens of one sequence (or one token of it, where a key that is not finite makes the pass be done over).  CTAs are persistent and take
// the grid's next one in their own stead (cluster launch control): an item's boxes are on their way while the last one's softmax, products and output
// run (with a CTA per 64 rows 12 us of 36 passed around its products).
//
// Bound: at M = 64 the tensor core runs at half rate, 2176 cycles a tile (measured: 32, 64, 128 cycles for N = 64, 128, 256; a thread's loop that works out
// descriptors and phases between products takes longer than that).  Its shared-memory reads and the boxes' writes take 1664.  Measured on B200, bf16, 16
// heads: four prompts of 2048 tokens 571 us with latent_attn_tc.cu -> 425 (688 TFLOP/s); at the clock that the power cap leaves (1.76 GHz in a loop of seconds)
// the products are two thirds of that.  32 heads, three ragged prompts of up to 1000 tokens at 1900, window 2048: 544 -> 382.
#include "latent_attn_tc.cuh"
#include "mma_helpers.cuh"
#include "tc_helpers.cuh"
#include "typed_io.cuh"

namespace sllm {

using namespace tc;

constexpr int LP_ROWS = 64, LP_KEYS = 64, LP_R = 512, LP_DR = 64, LP_D = LP_R + LP_DR, LP_CHUNKS = LP_D / 64;
constexpr int LP_THREADS = 512, LP_STAGES = 3, LP_BUFS = 3;                     // buffers of O_q
constexpr int LP_GROUP = LP_CHUNKS * 1024;             // bytes of 8 key rows: nine SWIZZLE_128B atoms
constexpr int LP_STAGE = 8 * LP_GROUP;
constexpr int LP_QCHUNK = 64 * 128;                    // queries on their way: [chunk][64 rows][128 B]
constexpr int LP_MISC = LP_STAGES * LP_STAGE;
constexpr int LP_CONSUMERS = 14;                       // warps that read an item: issuers, softmax, accumulators
constexpr int LP_Q_COL = 0, LP_S_COL = 288, LP_O_COL = 0, LP_P_COL = 384;       // S two of 64; O_q three of 128, P two of 32
constexpr float LP_LOG2E = 1.4426950408889634f;
constexpr int LP_REGS_FEW = 72, LP_REGS_SOFTMAX = 88, LP_REGS_O = 176;
static_assert(LP_REGS_FEW + LP_REGS_SOFTMAX + 2 * LP_REGS_O <= 4 * 128, "the warpgroups' shares must fit what the block was launched with");

struct LatentPromptBars {
    uint64_t full[LP_STAGES], empty[LP_STAGES], landed, q_full, next;
    uint64_t item_full[2], item_empty[2];
    uint64_t s_full[2], s_empty[2], p_full[2], p_empty[2], a_empty[2], f_full[2], f_empty[2];
    uint64_t o_full[LP_BUFS], o_empty[LP_BUFS];
};

__device__ __forceinline__ uint64_t lp_desc(uint64_t base, uint32_t low) { return (base & 0xffffffff00000000ull) | low; }

// Four words of each lane of a quad, w[k] for group k -> the four lanes' words of group lane % 4, in the lanes' order
__device__ __forceinline__ void lp_turn(uint32_t (&w)[4]) {
    const bool odd = threadIdx.x & 1, high = threadIdx.x & 2;
#pragma unroll
    for (int k = 0; k < 4; k += 2) {
        const uint32_t x = __shfl_xor_sync(0xffffffffu, odd ? w[k] : w[k + 1], 1);
        if (odd) w[k] = x;
        else w[k + 1] = x;
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const uint32_t x = __shfl_xor_sync(0xffffffffu, high ? w[k] : w[k + 2], 2);
        if (high) w[k] = x;
        else w[k + 2] = x;
    }
}

// What the warps of a CTA have to know of an item: tokens ts .. ts + n - 1 of one sequence at positions pos0 .., `tiles` tiles of keys from key0 on, of which
// see_lo .. see_hi are seen; solo >= 0: the item is for this token alone; mark: where it says that it met a key that is not finite
struct LpItem { int valid, ts, n, seq, pos0, key0, tiles, see_lo, see_hi, solo, h0, mark; };
constexpr int LP_MARKS = 32;                              // items between looks at the marks
struct LpShared {
    LatentPromptBars bars;
    uint32_t tmem;
    alignas(16) uint8_t answer[16];
    LpItem items[2], marked[LP_MARKS];
    volatile int tainted[LP_MARKS];
    float alpha[2][LP_ROWS], factor[2][LP_ROWS];          // [buffer][row]: what a tile's maximum leaves of O; 1 / sum, times the gate
};
constexpr int LP_SMEM = LP_MISC + sizeof(LpShared);
static_assert(LP_SMEM <= 227 * 1024, "");

template <typename T>
__global__ void __launch_bounds__(LP_THREADS, 1) latent_attn_prompt_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap qmap,
                                                                           const LatentTc p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    LpShared& sh = *reinterpret_cast<LpShared*>(smem + LP_MISC);
    LatentPromptBars* bars = &sh.bars;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hp = 1 << p.hp_log2;

    if (tid == 0) {
        for (int i = 0; i < LP_STAGES; i++) { mbar_init(smem_u32(&bars->full[i]), 1); mbar_init(smem_u32(&bars->empty[i]), 1); }
        for (int i = 0; i < 2; i++) {
            mbar_init(smem_u32(&bars->s_full[i]), 1); mbar_init(smem_u32(&bars->s_empty[i]), 128);
            mbar_init(smem_u32(&bars->p_full[i]), 128); mbar_init(smem_u32(&bars->p_empty[i]), 1);
            mbar_init(smem_u32(&bars->a_empty[i]), 8);
            mbar_init(smem_u32(&bars->f_full[i]), 128); mbar_init(smem_u32(&bars->f_empty[i]), 8);
            mbar_init(smem_u32(&bars->item_full[i]), 1); mbar_init(smem_u32(&bars->item_empty[i]), LP_CONSUMERS);
        }
        for (int i = 0; i < LP_BUFS; i++) { mbar_init(smem_u32(&bars->o_full[i]), 1); mbar_init(smem_u32(&bars->o_empty[i]), 128); }
        mbar_init(smem_u32(&bars->landed), 1); mbar_init(smem_u32(&bars->q_full), 128); mbar_init(smem_u32(&bars->next), 1);
        mbar_fence_init();
        tma_prefetch_desc(&map); tma_prefetch_desc(&qmap);
    }
    if (warp == 0) sh.tainted[lane] = 0;
    static_assert(LP_MARKS == 32, "a lane a mark");
    if (warp == 1) tmem_alloc<512>(smem_u32(&sh.tmem));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    wait_previous();
    launch_next();

    constexpr uint32_t UPPER = 16u << 16;                 // lanes 16 .. 31
    // Item n, as warp 0 has left it.  Every role counts ring entries (an item's queries, then its tiles) and tiles: the barriers' phases follow from them
    auto take = [&](int n) {
        mbar_wait(smem_u32(&bars->item_full[n & 1]), (n >> 1) & 1);
        const LpItem it = sh.items[n & 1];
        __syncwarp();
        return it;
    };
    auto done_with = [&](int n) { if (lane == 0) mbar_arrive(smem_u32(&bars->item_empty[n & 1])); };

    if (warp < 4) {
        reg_dec<LP_REGS_FEW>();
        if (warp == 0) {
            // ======================================================= items and boxes
            int e = 0, ragged_done = 0, items = 0, marks = 0, answers = 0;      // ring entries, phases of `landed`, ...
            auto first_seen = [&](int pos) { return p.window > 0 ? max(0, pos - p.window + 1) : 0; };
            // One item: it is made known, then its queries and its tiles are loaded
            auto run = [&](const LpItem& it, bool ask) {
                if (lane == 0) {
                    mbar_wait(smem_u32(&bars->item_empty[items & 1]), ((items >> 1) & 1) ^ 1);
                    sh.items[items & 1] = it;
                    mbar_arrive(smem_u32(&bars->item_full[items & 1]));
                }
                items++;
                __syncwarp();
                if (!it.valid) return;
                if (lane == 0) {
                    if (ask) ask_next_cta(smem_u32(sh.answer), smem_u32(&bars->next));
                    const int st = e % LP_STAGES;
                    mbar_wait(smem_u32(&bars->empty[st]), ((e / LP_STAGES) & 1) ^ 1);
                    mbar_arrive_expect_tx(smem_u32(&bars->full[st]), LP_R / 64 * LP_QCHUNK);
                    tma_load_4d(smem_u32(smem + st * LP_STAGE), &qmap, smem_u32(&bars->full[st]), 0, it.h0, it.ts, 0);
                }
                e++;
                const int* bt = p.block_table + (int64_t)it.seq * p.max_blocks_per_seq;
                const int hi = it.pos0 + it.n - 1;
                auto rows = [&](int j) {                  // group of eight cache rows at which the lane's box of tile j begins, -1: none
                    const int kp = it.key0 + j * LP_KEYS + 16 * lane;
                    if (lane >= 4 || j >= it.tiles || kp > hi) return -1;
                    const int b = kp / p.block_size;
                    return (int)((((int64_t)bt[b] * p.n_slots + p.slot) * p.block_size + (kp - b * p.block_size)) >> 3);
                };
                int next = rows(0);
                for (int j = 0; j < it.tiles; j++, e++) {
                    const int group = next, st = e % LP_STAGES, base = it.key0 + j * LP_KEYS;
                    next = rows(j + 1);
                    const bool ragged = base < it.see_lo || base + LP_KEYS - 1 > it.see_hi;
                    const uint32_t full = smem_u32(&bars->full[st]), bar = ragged ? smem_u32(&bars->landed) : full;
                    const int boxes = __popc(__ballot_sync(0xffffffffu, group >= 0));
                    if (lane == 0) {
                        mbar_wait(smem_u32(&bars->empty[st]), ((e / LP_STAGES) & 1) ^ 1);
                        mbar_arrive_expect_tx(bar, (uint32_t)boxes * 2 * LP_GROUP);
                    }
                    __syncwarp();
                    if (group >= 0) tma_load_4d(smem_u32(smem + st * LP_STAGE) + lane * 2 * LP_GROUP, &map, bar, 0, 0, 0, group);
                    if (!ragged) continue;
                    mbar_wait(bar, ragged_done++ & 1);    // rows that are not seen become zero
                    // four rows at a time, eight lanes to a row's 128 bytes of each chunk (a row at a time 200 cycles each: up to 7 us an item, which
                    // for short prompts is most of it; us, 64 of up to 60 tokens, 16 heads, 73.7 / 52.0, 200 of up to 100, 4 heads, 91.7 / 65.0)
                    for (int row = lane >> 3; row < LP_KEYS; row += 4) {
                        if (base + row >= it.see_lo && base + row <= it.see_hi) continue;
                        uint8_t* at = smem + st * LP_STAGE + (row >> 3) * LP_GROUP + (row & 7) * 128 + (lane & 7) * 16;
#pragma unroll
                        for (int c = 0; c < LP_CHUNKS; c++) *reinterpret_cast<uint4*>(at + c * 1024) = make_uint4(0, 0, 0, 0);
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full);
                }
            };
            // Items that met a key that is not finite among those that only some of their tokens see are done over, token by token
            auto look_back = [&]() {
                for (int i = max(0, items - 2); i < items; i++) mbar_wait(smem_u32(&bars->item_empty[i & 1]), (i >> 1) & 1);      // (softmax warps are done)
                const uint32_t bad = __ballot_sync(0xffffffffu, sh.tainted[lane] != 0 && lane < marks);
                __syncwarp();
                sh.tainted[lane] = 0;
                __syncwarp();
                for (int m = 0; m < marks; m++) {
                    if (!(bad >> m & 1)) continue;
                    LpItem it = sh.marked[m];
                    it.mark = -1;
                    for (it.solo = 0; it.solo < it.n; it.solo++) {
                        it.see_hi = it.pos0 + it.solo; it.see_lo = first_seen(it.see_hi);
                        run(it, false);
                    }
                }
                marks = 0;
            };
            bool asked = false;
            for (int bx = blockIdx.x, by = blockIdx.y, more = 1; more;) {
                const int t_first = (gridDim.x - 1 - bx) * p.qt, ntok = min(p.qt, p.num_tokens - t_first);      // a prompt's last tokens have the most keys: first
                LpItem it;
                it.valid = 1; it.solo = -1; it.h0 = by * hp;
                for (int i0 = 0; i0 < ntok; i0 += it.n) { // segments: runs of one sequence at consecutive positions
                    it.ts = t_first + i0;
                    const int left = ntok - i0, a = it.ts + min(lane, left - 1), b = it.ts + min(lane + 32, left - 1);
                    const int sa = p.tok_seq[a], sb = p.tok_seq[b], qa = p.tok_pos[a], qb = p.tok_pos[b];
                    it.seq = __shfl_sync(0xffffffffu, sa, 0); it.pos0 = __shfl_sync(0xffffffffu, qa, 0);
                    const uint32_t cut_a = __ballot_sync(0xffffffffu, lane >= left || sa != it.seq || qa != it.pos0 + lane);
                    const uint32_t cut_b = __ballot_sync(0xffffffffu, lane + 32 >= left || sb != it.seq || qb != it.pos0 + lane + 32);
                    it.n = cut_a ? __ffs(cut_a) - 1 : cut_b ? 31 + __ffs(cut_b) : 64;
                    it.see_hi = it.pos0 + it.n - 1; it.see_lo = first_seen(it.pos0);
                    it.key0 = it.see_lo & ~15;
                    it.tiles = (it.see_hi - it.key0) / LP_KEYS + 1;
                    if (marks == LP_MARKS) look_back();
                    it.mark = marks++;
                    if (lane == 0) sh.marked[it.mark] = it;
                    __syncwarp();
                    run(it, !asked);
                    asked = true;
                }
                mbar_wait(smem_u32(&bars->next), answers++ & 1);
                more = next_cta(smem_u32(sh.answer), bx, by);
                asked = false;
            }
            look_back();
            LpItem end;
            end.valid = 0;
            run(end, false);
        } else if (warp == 1) {
            // ======================================================= product issuers (the warps wait converged, one lane issues).  Descriptors differ in
            // their low words by constants
            constexpr uint32_t IDESC_S = make_instr_desc(LP_ROWS, LP_KEYS, UmmaFmt<T>::value, 0, 0);
            const uint64_t dk = make_smem_desc(smem_u32(smem), 16, LP_GROUP);
            for (int n = 0, e = 0, t = 0;; n++) {
                const LpItem item = take(n);
                done_with(n);
                if (!item.valid) break;
                mbar_wait(smem_u32(&bars->q_full), n & 1);
                if (lane == 0) mbar_arrive(smem_u32(&bars->empty[e % LP_STAGES]));      // the queries are in TMEM
                e++;
                for (int j = 0; j < item.tiles; j++, e++, t++) {
                    const int st = e % LP_STAGES, b = t & 1;
                    const uint32_t low = (uint32_t)dk + ((st * LP_STAGE) >> 4), s_addr = tmem + LP_S_COL + 64 * b;
                    mbar_wait(smem_u32(&bars->full[st]), (e / LP_STAGES) & 1);
                    mbar_wait(smem_u32(&bars->s_empty[b]), ((t >> 1) & 1) ^ 1);
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll 3
                        for (int c = 0; c < LP_CHUNKS; c++)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                umma_ts(s_addr, tmem + LP_Q_COL + 32 * c + 8 * k, lp_desc(dk, low + ((c * 1024 + k * 32) >> 4)), IDESC_S, c > 0 || k > 0 ? 1u : 0u);
                        umma_commit(smem_u32(&bars->s_full[b]));
                    }
                    __syncwarp();
                }
            }
        } else if (warp == 2) {
            constexpr uint32_t IDESC_O = make_instr_desc(LP_ROWS, 128, UmmaFmt<T>::value, 0, 1);
            const uint64_t dv = make_smem_desc(smem_u32(smem), 1024, LP_GROUP);
            for (int n = 0, e = 0, t = 0;; n++) {
                const LpItem item = take(n);
                done_with(n);
                if (!item.valid) break;
                e++;
                for (int j = 0; j < item.tiles; j++, e++, t++) {
                    const int st = e % LP_STAGES, b = t & 1;
                    const uint32_t low = (uint32_t)dv + ((st * LP_STAGE) >> 4), p_addr = tmem + UPPER + LP_P_COL + 32 * b;
                    mbar_wait(smem_u32(&bars->p_full[b]), (t >> 1) & 1);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int i = 4 * t + q, buf = i % LP_BUFS;
                        mbar_wait(smem_u32(&bars->o_empty[buf]), ((i / LP_BUFS) & 1) ^ 1);
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                umma_ts(tmem + UPPER + LP_O_COL + 128 * buf, p_addr + 8 * k, lp_desc(dv, low + ((2 * k * LP_GROUP + q * 2048) >> 4)), IDESC_O, k > 0 ? 1u : 0u);
                            umma_commit(smem_u32(&bars->o_full[buf]));
                            if (q == 3) { umma_commit(smem_u32(&bars->empty[st])); umma_commit(smem_u32(&bars->p_empty[b])); }
                        }
                        __syncwarp();
                    }
                }
            }
        }
    } else if (warp < 8) {
        reg_dec<LP_REGS_SOFTMAX>();
        const uint32_t tlane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        const int ra = 16 * (warp & 3) + (lane >> 2), rb = ra + 8, ja = ra >> p.hp_log2, jb = rb >> p.hp_log2;
        const float c = p.scale * LP_LOG2E;
        for (int n = 0, e = 0, t = 0;; n++) {
            const LpItem item = take(n);
            if (!item.valid) break;
            const int ha = item.h0 + (ra & (hp - 1)), hb = item.h0 + (rb & (hp - 1));
            const bool live_a = ja < item.n && ha < p.H, live_b = jb < item.n && hb < p.H;
            // ---- queries into TMEM (the scores of the items before have all been read): the rotated ones are asked for first and used last.  A word is
            // a pair of entries, pairs (2i, 2i + 1) below rot_dims turn
            {
                uint32_t w[16];                           // word 4 i + lane % 4 of row a (even) and b
                float2 cs[8];
                const int rhalf = p.rot_dims >> 1;
                auto angles = [&](int64_t tok) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int pair = 4 * i + (lane & 3);
                        cs[i] = pair < rhalf ? make_float2(p.cosb[tok * rhalf + pair], p.sinb[tok * rhalf + pair]) : make_float2(1.f, 0.f);
                    }
                };
                auto turn = [&](int r) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const float2 x = Traits<T>::to_f2(*reinterpret_cast<typename Traits<T>::T2*>(&w[2 * i + r]));
                        if (4 * i + (lane & 3) < rhalf) w[2 * i + r] = pack2<T>(x.x * cs[i].x - x.y * cs[i].y, x.y * cs[i].x + x.x * cs[i].y);
                    }
                };
                const int64_t tok_a = item.ts + (live_a ? ja : 0), tok_b = item.ts + (live_b ? jb : 0);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const bool live = r ? live_b : live_a;
                    const T* qr = reinterpret_cast<const T*>(p.q_rot) + (r ? tok_b : tok_a) * p.qr_st + (live ? (int64_t)(r ? hb : ha) * p.qr_sh : 0) + 2 * (lane & 3);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        if (p.rot_vec) w[2 * i + r] = *reinterpret_cast<const uint32_t*>(qr + 8 * i);
                        else w[2 * i + r] = (uint32_t)reinterpret_cast<const unsigned short*>(qr)[8 * i] | (uint32_t)reinterpret_cast<const unsigned short*>(qr)[8 * i + 1] << 16;
                    }
                }
                angles(tok_a);
                const int st = e % LP_STAGES;
                mbar_wait(smem_u32(&bars->full[st]), (e / LP_STAGES) & 1);
                tc_fence_after();
                const uint8_t* q_sm = smem + st * LP_STAGE;
#pragma unroll 1
                for (int ch = 0; ch < LP_R / 64; ch++) {
                    uint32_t v[16];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        v[2 * i] = *reinterpret_cast<const uint32_t*>(q_sm + ch * LP_QCHUNK + swizzled(ra, i) + 4 * (lane & 3));
                        v[2 * i + 1] = *reinterpret_cast<const uint32_t*>(q_sm + ch * LP_QCHUNK + swizzled(rb, i) + 4 * (lane & 3));
                    }
                    tmem_st_16x32(tlane + LP_Q_COL + 32 * ch, v);
                }
                turn(0);
                angles(tok_b);
                turn(1);
                tmem_st_16x32(tlane + LP_Q_COL + LP_R / 2, w);
                tmem_st_wait();
                tc_fence_before();
                fence_proxy_async();                      // boxes overwrite the stage
                mbar_arrive(smem_u32(&bars->q_full));
                e += 1 + item.tiles;
            }
            // ======================================================= softmax.  A row sees the keys first .. last (none in a dead row)
            const int last_a = live_a ? item.pos0 + ja : -1, last_b = live_b ? item.pos0 + jb : -1;
            const int first_a = p.window > 0 ? last_a - p.window + 1 : 0, first_b = p.window > 0 ? last_b - p.window + 1 : 0;
            const uint32_t size_a = live_a ? 0x7fffffffu : 0u, size_b = live_b ? 0x7fffffffu : 0u;
            float ma = -INFINITY, mb = -INFINITY, la = 0.f, lb = 0.f;
            if (p.sink != nullptr) {
                if (live_a) { ma = p.sink[ha] * LP_LOG2E; la = (lane & 3) == 0 ? 1.f : 0.f; }
                if (live_b) { mb = p.sink[hb] * LP_LOG2E; lb = (lane & 3) == 0 ? 1.f : 0.f; }
            }
            const bool all_live = item.n * hp >= LP_ROWS && item.h0 + hp <= p.H && p.window <= 0;
            uint32_t top = 0;                             // the largest magnitude (as bits) among the masked scores
            for (int j = 0; j < item.tiles; j++, t++) {
                const int b = t & 1;
                mbar_wait(smem_u32(&bars->s_full[b]), (t >> 1) & 1);
                tc_fence_after();
                uint32_t s[32];
                tmem_ld_16x64(tlane + LP_S_COL + 64 * b, s);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->s_empty[b]));
                const int base = item.key0 + j * LP_KEYS;
                if (base + LP_KEYS - 1 > item.pos0 || !all_live) {
                    const int cb = base + 2 * (lane & 3);
#pragma unroll
                    for (int i = 0; i < 8; i++)
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const int kp = cb + 8 * i + k;
                            if (kp > last_a || kp < first_a) { top = max(top, s[4 * i + k] & size_a); s[4 * i + k] = 0xff800000u; }
                            if (kp > last_b || kp < first_b) { top = max(top, s[4 * i + 2 + k] & size_b); s[4 * i + 2 + k] = 0xff800000u; }
                        }
                }
                float xa = -INFINITY, xb = -INFINITY;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    xa = max3(xa, __uint_as_float(s[4 * i]), __uint_as_float(s[4 * i + 1]));
                    xb = max3(xb, __uint_as_float(s[4 * i + 2]), __uint_as_float(s[4 * i + 3]));
                }
                xa = fmaxf(xa, __shfl_xor_sync(0xffffffffu, xa, 1)); xb = fmaxf(xb, __shfl_xor_sync(0xffffffffu, xb, 1));
                xa = fmaxf(xa, __shfl_xor_sync(0xffffffffu, xa, 2)); xb = fmaxf(xb, __shfl_xor_sync(0xffffffffu, xb, 2));
                const float na = fmaxf(ma, xa * c), nb = fmaxf(mb, xb * c);
                const bool need_a = na > ma, need_b = nb > mb;
                const float al_a = need_a ? fast_exp2_tc(ma - na) : 1.f, al_b = need_b ? fast_exp2_tc(mb - nb) : 1.f;
                if (need_a) { ma = na; la *= al_a; }
                if (need_b) { mb = nb; lb *= al_b; }
                const float sub_a = ma == -INFINITY ? 0.f : -ma, sub_b = mb == -INFINITY ? 0.f : -mb;      // nothing seen yet
                uint32_t w[16];                           // P in the storage type; the sums take the rounded values
#pragma unroll
                for (int i = 0; i < 16; i++) {            // two keys of row a (even i) or b
                    const float sub = i & 1 ? sub_b : sub_a;
                    const float p0 = fast_exp2_tc(fmaf(__uint_as_float(s[2 * i]), c, sub)), p1 = fast_exp2_tc(fmaf(__uint_as_float(s[2 * i + 1]), c, sub));
                    w[i] = pack2<T>(p0, p1);
                    const float2 f = Traits<T>::to_f2(*reinterpret_cast<typename Traits<T>::T2*>(&w[i]));
                    (i & 1 ? lb : la) += f.x + f.y;
                }
                mbar_wait(smem_u32(&bars->a_empty[b]), ((t >> 1) & 1) ^ 1);
                if ((lane & 3) == 0) { sh.alpha[b][ra] = al_a; sh.alpha[b][rb] = al_b; }
                mbar_wait(smem_u32(&bars->p_empty[b]), ((t >> 1) & 1) ^ 1);
                tc_fence_after();
                tmem_st_16x32(tlane + UPPER + LP_P_COL + 32 * b, w);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->p_full[b]));
            }
            la += __shfl_xor_sync(0xffffffffu, la, 1); la += __shfl_xor_sync(0xffffffffu, la, 2);
            lb += __shfl_xor_sync(0xffffffffu, lb, 1); lb += __shfl_xor_sync(0xffffffffu, lb, 2);
            // (a row whose sum is NaN is NaN by its own keys)
            if (item.mark >= 0 && item.n > 1 && top >= 0x7f800000u && ((live_a && la == la) || (live_b && lb == lb))) sh.tainted[item.mark] = 1;
            mbar_wait(smem_u32(&bars->f_empty[n & 1]), ((n >> 1) & 1) ^ 1);
            if ((lane & 3) == 0) {
                auto factor = [&](float l, bool live, int jj, int h) {
                    if (!live) return 0.f;
                    const float f = 1.f / l;
                    return p.gate == nullptr ? f : f * (1.f / (1.f + expf(-ldf(reinterpret_cast<const T*>(p.gate) + (int64_t)(item.ts + jj) * p.gate_st + h))));
                };
                sh.factor[n & 1][ra] = factor(la, live_a, ja, ha);
                sh.factor[n & 1][rb] = factor(lb, live_b, jb, hb);
            }
            mbar_arrive(smem_u32(&bars->f_full[n & 1]));
            __syncwarp();
            done_with(n);
        }
    } else {
        reg_inc<LP_REGS_O>();
        const int half = (warp - 8) >> 2, quad = warp & 3;                        // O_q of q = half, half + 2
        const uint32_t tlane = tmem + ((uint32_t)(32 * quad) << 16) + UPPER;
        const int ra = 16 * quad + (lane >> 2), rb = ra + 8;                      // rows 16 quad + lane / 4 and + 8
        for (int n = 0, t = 0;; n++) {
            const LpItem item = take(n);
            done_with(n);
            if (!item.valid) break;
            float2 acc[64];                               // [32 q + 2 i + r]: a pair of columns of row a or b in the i-th eight columns of the q-th O_q
#pragma unroll
            for (int i = 0; i < 64; i++) acc[i] = make_float2(0.f, 0.f);
            for (int j = 0; j < item.tiles; j++, t++) {
                const int b = t & 1;
                mbar_wait(smem_u32(&bars->p_full[b]), (t >> 1) & 1);
                const float fa = sh.alpha[b][ra], fb = sh.alpha[b][rb];
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars->a_empty[b]));
                const float2 f2[2] = {make_float2(fa, fa), make_float2(fb, fb)};
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int i = 4 * t + 2 * q + half, buf = i % LP_BUFS;
                    // (This half waits for every other phase of a buffer.  The one between, of product i - 3, is over: the products' warp issues one behind the
                    // other, and i - 2, which this half has waited for, came after it)
                    mbar_wait(smem_u32(&bars->o_full[buf]), (i / LP_BUFS) & 1);
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t v[32];
                        tmem_ld_16x64(tlane + LP_O_COL + 128 * buf + 64 * h, v);
                        tmem_ld_wait();
                        if (h == 1) {
                            tc_fence_before();
                            mbar_arrive(smem_u32(&bars->o_empty[buf]));
                        }
#pragma unroll
                        for (int k = 0; k < 16; k++) {
                            float2& x = acc[32 * q + 16 * h + k];
                            x = fma2(x, f2[k & 1], make_float2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1])));
                        }
                    }
                }
            }
            // ---- output
            mbar_wait(smem_u32(&bars->f_full[n & 1]), (n >> 1) & 1);
            const float fr[2] = {sh.factor[n & 1][ra], sh.factor[n & 1][rb]};
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->f_empty[n & 1]));
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int row = r ? rb : ra, jj = row >> p.hp_log2, h = item.h0 + (row & (hp - 1));
                const bool live = jj < item.n && h < p.H && (item.solo < 0 || jj == item.solo);
                const float f = fr[r];
                T* o = reinterpret_cast<T*>(p.out) + (int64_t)(item.ts + jj) * p.out_st + (int64_t)h * p.out_sh + 128 * half;
#pragma unroll
                for (int g = 0; g < 8; g++) {             // 32 columns at a time: the lane ends up with eight neighbouring ones
                    uint32_t w[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float2 x = acc[8 * g + 2 * k + r];
                        w[k] = pack2<T>(x.x * f, x.y * f);
                    }
                    lp_turn(w);
                    if (live) {
                        T* to = o + 256 * (g >> 2) + 32 * (g & 3) + 8 * (lane & 3);
                        if (p.out_vec) *reinterpret_cast<uint4*>(to) = make_uint4(w[0], w[1], w[2], w[3]);
                        else {
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const float2 x = Traits<T>::to_f2(*reinterpret_cast<typename Traits<T>::T2*>(&w[k]));
                                stf(to + 2 * k, x.x); stf(to + 2 * k + 1, x.y);
                            }
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc<512>(tmem);
}

// Where every SM has at least two and a half CTAs' rows to do (us, latent_attn_tc.cu / here, no window: 16 heads, one prompt of 1539 tokens 97 / 70, 40 of 38
// 38 / 29; 4 heads, two of 3078 163 / 142; 64 heads, two of 192 at 1500 175 / 125).  With fewer, few long segments end late here, where a CTA has taken its
// second before its first is done (4 heads, two of 1894, 240 CTAs, 71 / 80, two of 2486, 312 CTAs, 108 / 117; 16 heads, two of 473 30 / 32), though
// others gain (16 heads, 8 of 118 27 / 21).  Query views in which heads or tokens share their entries are left to latent_attn_tc.cu's plain loads.
bool latent_prompt_takes(const LatentTc& p, dim3 grid, int num_sms) {
    return 2ll * grid.x * grid.y >= 5ll * num_sms && p.r == LP_R && p.dr == LP_DR && p.block_size % 16 == 0 && p.nsplit == 1 && p.q_vec &&
           p.ql_st > 0 && p.ql_sh > 0 && get_tensor_map_encoder() != nullptr;
}

int launch_latent_attn_prompt(const LatentTc& p, dim3 grid, sllm_dtype_t dtype, cudaStream_t stream) {
    CUtensorMap map, qmap;
    const CUtensorMapDataType type = dtype == SLLM_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    auto encode = [&](CUtensorMap* m, const void* at, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
        const cuuint32_t es[4] = {1, 1, 1, 1};
        return get_tensor_map_encoder()(m, type, 4, const_cast<void*>(at), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    // (a block table names only blocks that there are: the map need not know how many)
    const cuuint64_t dims[4] = {64, 8, LP_CHUNKS, 1u << 28}, strides[3] = {LP_D * 2, 128, 8 * LP_D * 2};
    const cuuint32_t box[4] = {64, 8, LP_CHUNKS, 2};
    // queries: (64 d | heads | tokens | chunks); heads past the last are zero
    const cuuint64_t qdims[4] = {64, (cuuint64_t)p.H, (cuuint64_t)p.num_tokens, LP_R / 64};
    const cuuint64_t qstrides[3] = {(cuuint64_t)p.ql_sh * 2, (cuuint64_t)p.ql_st * 2, 128};
    const cuuint32_t qbox[4] = {64, 1u << p.hp_log2, (cuuint32_t)p.qt, LP_R / 64};
    if (encode(&map, p.cache, dims, strides, box) != CUDA_SUCCESS || encode(&qmap, p.q_lat, qdims, qstrides, qbox) != CUDA_SUCCESS) return -1;
    SLLM_DISPATCH_DTYPE(dtype, {
        static unsigned long long configured = 0;
        if (first_use_on_this_device(configured)) {
            const cudaError_t e = cudaFuncSetAttribute(latent_attn_prompt_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, LP_SMEM);
            SLLM_REQUIRE(e == cudaSuccess, "latent_attention: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        }
        launch_early(latent_attn_prompt_kernel<T>, grid, LP_THREADS, LP_SMEM, stream, map, qmap, p);
    });
    return check_launch("latent_attention (prompt rows)");
}

}  // namespace sllm
