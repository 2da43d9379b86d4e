// Latent attention for 16-bit storage on the fifth-generation tensor cores (tcgen05 + TMEM): the same function as latent_attn.cu, whose
// head comment gives the definition and the cache layout.
//
// A CTA owns up to 64 query ROWS: row = (token, head) with the heads of a token padded to a power of two, so 16 heads give four
// consecutive tokens of a prompt portion a common pass over their keys, and a decoded token's heads fill what they can of one pass.
// Tokens are walked in segments (runs of one sequence at consecutive positions), so any order of rows is correct.
//   S[64, 64 keys]  = Q K^T        M = 64, N = 64, D / 16 steps; Q and K in shared memory (K-major)
//   O[64, r]       += P K[:, :r]   M = 64, N = 256 twice; P from TMEM, the SAME key tile (now MN-major: a latent is key and value at once)
// Accumulators and P stay in TMEM: an M = 64 operand fills 16 of every 32 lanes, so the two halves of O lie in the same 256 columns (lane
// offsets 0 and 16); P (16-bit, two buffers) is written to both lane offsets, because an A operand lies in its accumulator's lanes; S has
// two buffers beside them.  The reference of the exponentials is the running maximum itself: a reference that trails it (by up to 2^8, say)
// would save most rescales of O (490 instead of 580 us below), but then the largest weight is not 1 and takes a rounding as well,
// 2.15e-3 instead of 2.01e-3 off 64-bit arithmetic in bf16.
//
// Single tokens of at most 16 heads fill one warp's 16 rows.  The next warp's rows repeat them and take as P what the rounding of the first
// left over, at no further product: weights of 8 and 8 bits (bf16).  With one rounding, fewer key splits (each rounds against its own
// maximum) cost precision: 64 tokens at 2048 keys 1.919e-3 off 64 bits in four splits of the mma.sync kernel, 1.945e-3 in two, now 1.791e-3.
//
// Shared memory is what decides the shape: 64 rows of Q (576 entries: 72 KiB) and two stages of 64 keys (72 KiB each) fill it.  A stage
// therefore is handed back in two pieces, each as soon as the product that reads it last is done: the first 256 columns after the first
// half of O, the rest after the second; producer warps gather each piece through the block table by cp.async (rows past the last
// visible key are zero).
//
// A weight of exactly 0 times a key row that is not finite is NaN, so a key that one row of a pass sees and another does not may reach both.
// Key and value are one row: a masked score that is not finite gives such a key away, and the segment is then done over, token by token,
// with the keys that the token does not see left zero (same tiles, same key splits).  A result depends on its own keys only.
//
// Bound: at M = 64 the tensor core runs at half rate, (D + r) * 64 * 64 multiply-adds per tile = 2176 cycles at D = 576, r = 512, and
// S's operands are 4 KiB of shared memory per 32 cycles; a decoded token is bound by its rows' bytes.  Measured on B200, bf16, 16 heads,
// r = 512: four prompts of 2048 tokens 3214 us with the mma.sync kernel of latent_attn.cu -> 573 us (509 TFLOP/s; large launches of
// such rows now run latent_attn_prompt.cu, 450 us); 64 decoded tokens at 2048 keys 88 -> 49 us with the merge.
#include "latent_attn_tc.cuh"
#include "mma_helpers.cuh"
#include "tc_helpers.cuh"
#include "typed_io.cuh"

namespace sllm {

using namespace tc;

constexpr int LT_ROWS = 64, LT_KEYS = 64;
constexpr int LT_PW = 4;                            // producer warps per piece of a stage
constexpr int LT_MMA_WARP = 4 + 2 * LT_PW;          // warps 0-3 softmax and output, then the producers, then the product issuer
constexpr int LT_THREADS = (LT_MMA_WARP + 1) * 32;
constexpr int LT_CHUNK = 64 * 128;                  // bytes of 64 rows x 64 columns (SWIZZLE_128B atoms of 8 rows)
constexpr int LT_MAX_CHUNKS = 9;
constexpr int LT_STAGE = LT_MAX_CHUNKS * LT_CHUNK;
constexpr int LT_SMEM = 3 * LT_STAGE + 1024;
constexpr int LT_REST_PITCH = 512 + 4;              // floats of a row on its way from rows 16 .. 31 to rows 0 .. 15: O, then the sum
constexpr int LT_S_COL = 256, LT_P_COL = 384;       // TMEM columns: O 0..255, S two of 64, P two of 32
constexpr float LT_LOG2E = 1.4426950408889634f, LT_LN2 = 0.6931471805599453f;

struct LatentTcBars {
    uint64_t full[2][2], empty[2][2];                // [stage][piece]
    uint64_t s_full[2], s_empty[2], p_full[2], o_done[2];
};

// FULL: r = 512 and dr = 64, known to the compiler (the producers' and the issuer's loops are bound by their instructions).  ROWS: prompt
// rows (and single tokens of more heads); LT_SINGLES: single tokens of at most 16 heads, whose rows 16 .. 31 repeat rows 0 .. 15; LT_SHARED: prompt
// rows of a launch that leaves SMs over, whose CTAs of the same tokens take one segment each (in the first kernel this costs 3 %)
enum LatentRows { LT_PROMPTS, LT_SINGLES, LT_SHARED };
template <typename T, bool FULL, LatentRows ROWS>
__global__ void __launch_bounds__(LT_THREADS, 1) latent_attn_tc_kernel(const LatentTc p) {
    constexpr bool DUP = ROWS == LT_SINGLES;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* q_sm = smem;                            // [chunk][64 rows][128 B]
    uint8_t* k_sm = smem + LT_STAGE;                 // [stage][chunk][64 keys][128 B]
    LatentTcBars* bars = reinterpret_cast<LatentTcBars*>(smem + 3 * LT_STAGE);
    uint32_t* tmem_s = reinterpret_cast<uint32_t*>(smem + 3 * LT_STAGE + 512);
    volatile int* tainted = reinterpret_cast<int*>(tmem_s + 1);      // the last pass over a segment that met such a key
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int r = FULL ? 512 : p.r, dr = FULL ? 64 : p.dr, D = r + dr;
    const int n0 = r < 256 ? r : 256, n1 = r - n0;   // columns of O in its two halves
    const int c0 = n0 >> 6, chunks = (D + 63) >> 6;  // chunks of the first piece, of a row
    const int hp = 1 << p.hp_log2, h0 = blockIdx.y * hp;
    auto split = [&] { return (int)(ROWS == LT_SHARED ? blockIdx.z % p.nsplit : blockIdx.z); };      // (found where it is used)
    int t_first = (gridDim.x - 1 - blockIdx.x) * p.qt;            // the last tokens of a prompt have the most keys: first
    int ntok = min(p.qt, p.num_tokens - t_first);
    if constexpr (ROWS == LT_SHARED) {               // one segment each, the last CTA what is left
        wait_previous();
        auto length = [&](int left) {                // tokens of the segment at t_first
            const int a = t_first + min(lane, left - 1), b = t_first + min(lane + 32, left - 1);
            const int sa = p.tok_seq[a], sb = p.tok_seq[b], qa = p.tok_pos[a], qb = p.tok_pos[b];
            const int seq = __shfl_sync(0xffffffffu, sa, 0), pos = __shfl_sync(0xffffffffu, qa, 0);
            const uint32_t cut_a = __ballot_sync(0xffffffffu, lane >= left || sa != seq || qa != pos + lane);
            const uint32_t cut_b = __ballot_sync(0xffffffffu, lane + 32 >= left || sb != seq || qb != pos + lane + 32);
            return cut_a ? __ffs(cut_a) - 1 : cut_b ? 31 + __ffs(cut_b) : 64;
        };
        for (int k = blockIdx.z / p.nsplit; k > 0 && ntok > 0; k--) {
            const int n = length(ntok);
            t_first += n; ntok -= n;
        }
        if (blockIdx.z + p.nsplit < gridDim.z && ntok > 0) ntok = length(ntok);
    }
    auto head_row = [&](int row) { return DUP && row < 32 ? row & 15 : row; };      // the row whose token and head it is

    if (tid == 0) {
        *tainted = 0;
        for (int s = 0; s < 2; s++) {
            for (int g = 0; g < 2; g++) { mbar_init(smem_u32(&bars->full[s][g]), LT_PW); mbar_init(smem_u32(&bars->empty[s][g]), 1); }
            mbar_init(smem_u32(&bars->s_full[s]), 1); mbar_init(smem_u32(&bars->s_empty[s]), 128);
            mbar_init(smem_u32(&bars->p_full[s]), 128); mbar_init(smem_u32(&bars->o_done[s]), 1);
        }
        mbar_fence_init();
    }
    if (warp == LT_MMA_WARP) tmem_alloc<512>(smem_u32(tmem_s));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_s;
    wait_previous();
    // A merge of splits begins as the CTAs end: they leave no registers for its CTAs, which would all gather on the idle SMs (16 decoded tokens at
    // up to 4000, 16 heads: 29 us, launched earlier 36; the merge behind the launch's end 29, alone 31 instead of 30)
    if (p.nsplit == 1) launch_next();

    int n_done = 0;                                  // tiles of the passes before: every barrier's phase follows from it
    int pass = 0, solo = -1;                         // solo >= 0: the pass is for this token of the segment alone
    for (int i0 = 0; i0 < ntok;) {
        // ---- the segment: tokens ts .. ts + n - 1 of one sequence at positions pos0 ..; its keys lo .. hi, this CTA's tiles of them
        const int ts = t_first + i0, left = ntok - i0;
        int n, seq, pos0;
        {
            const int a = ts + min(lane, left - 1), b = ts + min(lane + 32, left - 1);
            const int sa = p.tok_seq[a], sb = p.tok_seq[b], qa = p.tok_pos[a], qb = p.tok_pos[b];
            seq = __shfl_sync(0xffffffffu, sa, 0); pos0 = __shfl_sync(0xffffffffu, qa, 0);
            const uint32_t cut_a = __ballot_sync(0xffffffffu, lane >= left || sa != seq || qa != pos0 + lane);
            const uint32_t cut_b = __ballot_sync(0xffffffffu, lane + 32 >= left || sb != seq || qb != pos0 + lane + 32);
            n = cut_a ? __ffs(cut_a) - 1 : cut_b ? 31 + __ffs(cut_b) : 64;
        }
        pass++;
        const int* bt = p.block_table + (int64_t)seq * p.max_blocks_per_seq;
        const int hi = pos0 + n - 1;
        const int lo = (p.window > 0 && pos0 - p.window + 1 > 0) ? pos0 - p.window + 1 : 0;
        const int all = (hi - lo) / LT_KEYS + 1, per = (all + p.nsplit - 1) / p.nsplit;
        const int tile0 = min(all, split() * per), ntiles = min(all, tile0 + per) - tile0;
        const int key0 = lo + tile0 * LT_KEYS;
        const int see_hi = solo < 0 ? hi : pos0 + solo;                        // keys outside are left zero
        const int see_lo = solo < 0 || p.window <= 0 ? lo : max(lo, pos0 + solo - p.window + 1);

        // producers: piece g of every tile, rows r0 .. r0 + 64 / LT_PW - 1; eight lanes a 128-byte row piece
        const bool producer = warp >= 4 && warp < LT_MMA_WARP;
        const int g = (warp - 4) / LT_PW, r0 = (64 / LT_PW) * ((warp - 4) % LT_PW), piece = lane & 7;
        auto key_row = [&](int j) {                  // cache row of key r0 + lane of tile j, -1 for one that is not visible
            const int kp = key0 + j * LT_KEYS + r0 + lane;
            if (lane >= 64 / LT_PW || kp > see_hi || kp < see_lo) return -1ll;
            const int b = kp / p.block_size;
            return ((long long)bt[b] * p.n_slots + p.slot) * p.block_size + (kp - b * p.block_size);
        };
        auto load = [&](int st, long long rowi) {
#pragma unroll
            for (int i = 0; i < 16 / LT_PW; i++) {
                const int row = r0 + 4 * i + (lane >> 3);
                const long long ri = __shfl_sync(0xffffffffu, rowi, 4 * i + (lane >> 3));
                const int bytes = ri >= 0 ? 16 : 0;
                const T* src = reinterpret_cast<const T*>(p.cache) + (ri >= 0 ? ri * D + piece * 8 : 0);
                const uint32_t dst = smem_u32(k_sm + st * LT_STAGE) + swizzled(row, piece);
                if constexpr (FULL) {
                    if (g == 0) {
#pragma unroll
                        for (int c = 0; c < 4; c++) cp_async16(dst + c * LT_CHUNK, src + c * 64, bytes);
                    } else {
#pragma unroll
                        for (int c = 4; c < 9; c++) cp_async16(dst + c * LT_CHUNK, src + c * 64, bytes);
                    }
                } else {
                    for (int c = g == 0 ? 0 : c0; c < (g == 0 ? c0 : chunks); c++)
                        if (c * 64 + piece * 8 < D) cp_async16(dst + c * LT_CHUNK, bytes ? src + c * 64 : src, bytes);
                }
            }
            cp_async_commit();
        };
        long long next = -1;
        if (producer && ntiles > 0) {                // the first tile's rows are on their way while the queries are staged
            const long long first = key_row(0);
            if (ntiles > 1) next = key_row(1);
            mbar_wait(smem_u32(&bars->empty[n_done & 1][g]), ((n_done >> 1) & 1) ^ 1);
            load(n_done & 1, first);
        }
        // ---- queries: [q_lat | rotated q_rot], zeros in rows without a (token, head).  The rotated entries (eight at a time; pairs
        // (2i, 2i + 1) below rot_dims turn) and their angles are asked for first and used last
        {
            const int half = p.rot_dims >> 1, eighths = dr >> 3;
            constexpr int AT_ONCE = (LT_ROWS * 8 + LT_THREADS - 1) / LT_THREADS;
            Vec8<T> u[AT_ONCE];
            float4 c4[AT_ONCE], s4[AT_ONCE];
#pragma unroll
            for (int b = 0; b < AT_ONCE; b++) {
                const int i = tid + b * LT_THREADS, row = eighths > 0 ? i / eighths : LT_ROWS, d = (i - row * eighths) * 8;
                const int j = head_row(row) >> p.hp_log2, h = h0 + (head_row(row) & (hp - 1));
                c4[b] = make_float4(1.f, 1.f, 1.f, 1.f); s4[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (p.rot_vec && row < LT_ROWS && j < n && h < p.H) {
                    u[b] = ld_vec8(reinterpret_cast<const T*>(p.q_rot) + (int64_t)(ts + j) * p.qr_st + (int64_t)h * p.qr_sh + d);
                    if (d < p.rot_dims) {
                        const int64_t ang = (int64_t)(ts + j) * half + (d >> 1);
                        c4[b] = *reinterpret_cast<const float4*>(p.cosb + ang); s4[b] = *reinterpret_cast<const float4*>(p.sinb + ang);
                    }
                }
            }
#pragma unroll 1
            for (int row = warp; row < LT_ROWS; row += LT_THREADS / 32) {
                const int j = head_row(row) >> p.hp_log2, h = h0 + (head_row(row) & (hp - 1));
                const bool live = j < n && h < p.H;
                const T* ql = reinterpret_cast<const T*>(p.q_lat) + (live ? (int64_t)(ts + j) * p.ql_st + (int64_t)h * p.ql_sh : 0);
                for (int c = lane; c < (r >> 3); c += 32) {
                    uint8_t* dst = q_sm + (c >> 3) * LT_CHUNK + swizzled(row, c & 7);
                    if (p.q_vec) {
                        cp_async16(smem_u32(dst), live ? ql + 8 * c : ql, live ? 16 : 0);
                    } else {
                        uint4 v = make_uint4(0, 0, 0, 0);
                        T* e = reinterpret_cast<T*>(&v);
                        if (live) {
#pragma unroll
                            for (int k = 0; k < 8; k++) e[k] = ql[8 * c + k];
                        }
                        *reinterpret_cast<uint4*>(dst) = v;
                    }
                }
            }
            cp_async_commit();
#pragma unroll
            for (int b = 0; b < AT_ONCE; b++) {
                const int i = tid + b * LT_THREADS, row = eighths > 0 ? i / eighths : LT_ROWS, d = (i - row * eighths) * 8;
                if (row >= LT_ROWS) continue;
                const int j = head_row(row) >> p.hp_log2, h = h0 + (head_row(row) & (hp - 1));
                const int64_t t = ts + j;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (j < n && h < p.H) {
                    float x[8], cs[4] = {c4[b].x, c4[b].y, c4[b].z, c4[b].w}, sn[4] = {s4[b].x, s4[b].y, s4[b].z, s4[b].w};
                    if (p.rot_vec) {
#pragma unroll
                        for (int e = 0; e < 4; e++) { const float2 f = Traits<T>::to_f2(u[b].v[e]); x[2 * e] = f.x; x[2 * e + 1] = f.y; }
                    } else {
                        const T* qr = reinterpret_cast<const T*>(p.q_rot) + t * p.qr_st + (int64_t)h * p.qr_sh + d;
                        const int64_t ang = t * half + (d >> 1);
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            x[2 * e] = ldf(qr + 2 * e); x[2 * e + 1] = ldf(qr + 2 * e + 1);
                            if (d + 2 * e < p.rot_dims) { cs[e] = p.cosb[ang + e]; sn[e] = p.sinb[ang + e]; }
                        }
                    }
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const bool turns = d + 2 * e < p.rot_dims;
                        const float a = x[2 * e], b2 = x[2 * e + 1];
                        w[e] = turns ? pack2<T>(a * cs[e] - b2 * sn[e], b2 * cs[e] + a * sn[e]) : pack2<T>(a, b2);
                    }
                    v = make_uint4(w[0], w[1], w[2], w[3]);
                }
                const int col = r + d;
                *reinterpret_cast<uint4*>(q_sm + (col >> 6) * LT_CHUNK + swizzled(row, (col & 63) >> 3)) = v;
            }
            cp_async_wait<0>();
            fence_proxy_async();
            __syncthreads();
        }

        if (producer) {
            for (int j = 0; j < ntiles; j++) {
                const int it = n_done + j, st = it & 1;
                if (j > 0) {                         // tile 0 has landed with the queries
                    const long long now = next;
                    if (j + 1 < ntiles) next = key_row(j + 1);
                    mbar_wait(smem_u32(&bars->empty[st][g]), ((it >> 1) & 1) ^ 1);
                    load(st, now);
                    cp_async_wait<0>();
                    fence_proxy_async();
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive(smem_u32(&bars->full[st][g]));
            }
        } else if (warp == LT_MMA_WARP) {
            // ======================================================= product issuer (the warp polls converged, one lane issues)
            const uint32_t idesc_s = make_instr_desc(LT_ROWS, LT_KEYS, UmmaFmt<T>::value, 0, 0);
            const uint32_t idesc_o0 = make_instr_desc(LT_ROWS, n0, UmmaFmt<T>::value, 0, 1);
            const uint32_t idesc_o1 = make_instr_desc(LT_ROWS, n1 > 0 ? n1 : 64, UmmaFmt<T>::value, 0, 1);
            const uint64_t dq = make_smem_desc(smem_u32(q_sm), 16, 1024), dk = make_smem_desc(smem_u32(k_sm), 16, 1024);
            const uint64_t dv = make_smem_desc(smem_u32(k_sm), LT_CHUNK, 1024);
            const int steps = D >> 4;
            constexpr uint32_t hi16 = 16u << 16;     // lane offset of the second half
            int js = 0, jp = 0;
            bool first_half = false;                 // the first piece's part of S(js) has been issued
            uint32_t spins = 0;
            while (jp < ntiles) {
                bool progressed = false;
                if (jp < js) {
                    const int it = n_done + jp, st = it & 1;
                    if (__all_sync(0xffffffffu, mbar_test_wait(smem_u32(&bars->p_full[st]), (it >> 1) & 1))) {
                        tc_fence_after();
                        if (elect_one()) {
                            const uint64_t vd = dv + (uint64_t)((st * LT_STAGE) >> 4);
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                umma_ts(tmem, tmem + LT_P_COL + 32 * st + 8 * k, vd + (uint64_t)((k * 2048) >> 4), idesc_o0, (jp > 0 || k > 0) ? 1u : 0u);
                            umma_commit(smem_u32(&bars->empty[st][0]));
                            if (n1 > 0) {
#pragma unroll
                                for (int k = 0; k < 4; k++)
                                    umma_ts(tmem + hi16, tmem + hi16 + LT_P_COL + 32 * st + 8 * k, vd + (uint64_t)((4 * LT_CHUNK + k * 2048) >> 4), idesc_o1,
                                            (jp > 0 || k > 0) ? 1u : 0u);
                            }
                            umma_commit(smem_u32(&bars->empty[st][1]));
                            umma_commit(smem_u32(&bars->o_done[st]));
                        }
                        __syncwarp();
                        jp++;
                        progressed = true;
                    }
                }
                if (js < ntiles) {
                    const int it = n_done + js, st = it & 1;
                    const uint32_t par = (it >> 1) & 1;
                    const uint32_t s_addr = tmem + LT_S_COL + 64 * st;
                    const uint64_t kd = dk + (uint64_t)((st * LT_STAGE) >> 4);
                    if (!first_half) {
                        const bool ready = mbar_test_wait(smem_u32(&bars->full[st][0]), par) && mbar_test_wait(smem_u32(&bars->s_empty[st]), par ^ 1);
                        if (__all_sync(0xffffffffu, ready)) {
                            tc_fence_after();
                            if (elect_one()) {
#pragma unroll 1
                                for (int k = 0; k < c0; k++) {
                                    const uint64_t off = (uint64_t)((k * LT_CHUNK) >> 4);
#pragma unroll
                                    for (int e = 0; e < 4; e++) umma_ss(s_addr, dq + off + 2 * e, kd + off + 2 * e, idesc_s, (k > 0 || e > 0) ? 1u : 0u);
                                }
                            }
                            __syncwarp();
                            first_half = progressed = true;
                        }
                    }
                    if (first_half && __all_sync(0xffffffffu, mbar_test_wait(smem_u32(&bars->full[st][1]), par))) {
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll 1
                            for (int k = c0; k < chunks; k++) {
                                const uint64_t off = (uint64_t)((k * LT_CHUNK) >> 4);
#pragma unroll
                                for (int e = 0; e < 4; e++)
                                    if (4 * k + e < steps) umma_ss(s_addr, dq + off + 2 * e, kd + off + 2 * e, idesc_s, 1);
                            }
                            umma_commit(smem_u32(&bars->s_full[st]));
                        }
                        __syncwarp();
                        first_half = false;
                        js++;
                        progressed = true;
                    }
                }
                if (progressed) spins = 0;
                else if (++spins > (1u << 24)) {
                    if (lane == 0) printf("sllm: latent attention watchdog (block %d,%d,%d js=%d jp=%d)\n", blockIdx.x, blockIdx.y, blockIdx.z, js, jp);
                    __trap();
                }
            }
        } else {
            // ======================================================= softmax: rows 16 w + lane / 4 (a) and + 8 (b), four lanes a row
            const int ra = 16 * warp + (lane >> 2), rb = ra + 8;
            const int ja = head_row(ra) >> p.hp_log2, jb = head_row(rb) >> p.hp_log2;
            const int ha = h0 + (head_row(ra) & (hp - 1)), hb = h0 + (head_row(rb) & (hp - 1));
            const bool rest = DUP && warp == 1;      // P is what the rounding of rows 0 .. 15 left over
            const bool live_a = ja < n && ha < p.H, live_b = jb < n && hb < p.H;
            // a row sees the keys first .. last (none in a dead row)
            const int last_a = live_a ? pos0 + ja : -1, last_b = live_b ? pos0 + jb : -1;
            const int first_a = p.window > 0 ? last_a - p.window + 1 : 0, first_b = p.window > 0 ? last_b - p.window + 1 : 0;
            const float c = p.scale * LT_LOG2E;
            float ma = -INFINITY, mb = -INFINITY, la = 0.f, lb = 0.f;
            if (p.sink != nullptr && split() == 0) {                        // the sink counts in ONE key split
                if (live_a) { ma = p.sink[ha] * LT_LOG2E; la = (lane & 3) == 0 && !rest ? 1.f : 0.f; }
                if (live_b) { mb = p.sink[hb] * LT_LOG2E; lb = (lane & 3) == 0 && !rest ? 1.f : 0.f; }
            }
            const uint32_t tlane = tmem + ((uint32_t)(32 * warp) << 16);
            // the row whose part of O this lane owns (lanes 16.. : its second half), and the lane that holds the row's state
            const int orow = lane & 15, from = 4 * (orow & 7);
            uint32_t top = 0;                        // the largest magnitude (as bits) among the masked scores
            for (int j = 0; j < ntiles; j++) {
                const int it = n_done + j, st = it & 1;
                mbar_wait(smem_u32(&bars->s_full[st]), (it >> 1) & 1);
                tc_fence_after();
                uint32_t s[32];
                tmem_ld_16x64(tlane + LT_S_COL + 64 * st, s);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->s_empty[st]));
                const int base = key0 + j * LT_KEYS;
                if (base + LT_KEYS - 1 > pos0 || p.window > 0 || n * hp < LT_ROWS || h0 + hp > p.H) {
                    const int cb = base + 2 * (lane & 3);
#pragma unroll
                    for (int i = 0; i < 8; i++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const int kp = cb + 8 * i + e;
                            if (kp > last_a || kp < first_a) { if (!DUP) top = max(top, s[4 * i + e] & 0x7fffffffu); s[4 * i + e] = 0xff800000u; }
                            if (kp > last_b || kp < first_b) { if (!DUP) top = max(top, s[4 * i + 2 + e] & 0x7fffffffu); s[4 * i + 2 + e] = 0xff800000u; }
                        }
                }
                float xa = -INFINITY, xb = -INFINITY;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    xa = fmaxf(xa, fmaxf(__uint_as_float(s[4 * i]), __uint_as_float(s[4 * i + 1])));
                    xb = fmaxf(xb, fmaxf(__uint_as_float(s[4 * i + 2]), __uint_as_float(s[4 * i + 3])));
                }
                xa = fmaxf(xa, __shfl_xor_sync(0xffffffffu, xa, 1)); xa = fmaxf(xa, __shfl_xor_sync(0xffffffffu, xa, 2));
                xb = fmaxf(xb, __shfl_xor_sync(0xffffffffu, xb, 1)); xb = fmaxf(xb, __shfl_xor_sync(0xffffffffu, xb, 2));
                const float na = fmaxf(ma, xa * c), nb = fmaxf(mb, xb * c);
                const bool need_a = na > ma, need_b = nb > mb;
                const float al_a = need_a ? fast_exp2_tc(ma - na) : 1.f, al_b = need_b ? fast_exp2_tc(mb - nb) : 1.f;
                if (need_a) { ma = na; la *= al_a; }
                if (need_b) { mb = nb; lb *= al_b; }
                const float sub_a = ma == -INFINITY ? 0.f : -ma, sub_b = mb == -INFINITY ? 0.f : -mb;      // nothing seen yet
                uint32_t w[16];                      // P in the storage type; the sums take the rounded values
#pragma unroll
                for (int i = 0; i < 16; i++) {       // two keys of row a (even i) or b
                    const float sub = i & 1 ? sub_b : sub_a;
                    const float p0 = fast_exp2_tc(fmaf(__uint_as_float(s[2 * i]), c, sub)), p1 = fast_exp2_tc(fmaf(__uint_as_float(s[2 * i + 1]), c, sub));
                    w[i] = pack2<T>(p0, p1);
                    float2 f = Traits<T>::to_f2(*reinterpret_cast<typename Traits<T>::T2*>(&w[i]));
                    if (DUP && rest) {
                        w[i] = pack2<T>(p0 - f.x, p1 - f.y);
                        f = Traits<T>::to_f2(*reinterpret_cast<typename Traits<T>::T2*>(&w[i]));
                    }
                    (i & 1 ? lb : la) += f.x + f.y;
                }
                // P's buffer was last read by the products of tile j - 2; a rescale needs those of tile j - 1 to be done
                const bool rescale = j > 0 && __any_sync(0xffffffffu, need_a || need_b);
                if (rescale) mbar_wait(smem_u32(&bars->o_done[st ^ 1]), ((it - 1) >> 1) & 1);
                else if (j > 1) mbar_wait(smem_u32(&bars->o_done[st]), ((it >> 1) & 1) ^ 1);
                tc_fence_after();
                if (rescale) {
                    const float f0 = __shfl_sync(0xffffffffu, al_a, from), f1 = __shfl_sync(0xffffffffu, al_b, from);
                    const float f = orow < 8 ? f0 : f1;
#pragma unroll 1
                    for (int cc = 0; cc < n0; cc += 64) {      // n0 is in whole 64-column chunks
                        uint32_t o0[32], o1[32];
                        tmem_ld32(tlane + cc, o0);
                        tmem_ld32(tlane + cc + 32, o1);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; e++) {
                            o0[e] = __float_as_uint(__uint_as_float(o0[e]) * f);
                            o1[e] = __float_as_uint(__uint_as_float(o1[e]) * f);
                        }
                        tmem_st32(tlane + cc, o0);
                        tmem_st32(tlane + cc + 32, o1);
                    }
                }
                tmem_st_16x32(tlane + LT_P_COL + 32 * st, w);
                tmem_st_16x32(tlane + (16u << 16) + LT_P_COL + 32 * st, w);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->p_full[st]));
            }
            // ---- output: the lane owns row orow, columns n0 * (lane / 16) ..
            la += __shfl_xor_sync(0xffffffffu, la, 1); la += __shfl_xor_sync(0xffffffffu, la, 2);
            lb += __shfl_xor_sync(0xffffffffu, lb, 1); lb += __shfl_xor_sync(0xffffffffu, lb, 2);
            const float l0 = __shfl_sync(0xffffffffu, la, from), l1 = __shfl_sync(0xffffffffu, lb, from);
            const float m0 = __shfl_sync(0xffffffffu, ma, from), m1 = __shfl_sync(0xffffffffu, mb, from);
            const float m = orow < 8 ? m0 : m1;
            float l = orow < 8 ? l0 : l1;
            // (a row whose sum is NaN is NaN by its own keys)
            if (!DUP && solo < 0 && n > 1 && top >= 0x7f800000u && ((live_a && la == la) || (live_b && lb == lb))) *tainted = pass;
            const int row = head_row(16 * warp + orow), jj = row >> p.hp_log2, h = h0 + (row & (hp - 1));
            const bool live = jj < n && h < p.H && (solo < 0 || jj == solo);
            float* xs = reinterpret_cast<float*>(q_sm) + orow * LT_REST_PITCH;      // (the queries are done with)
            const int64_t t = ts + jj;
            const int col0 = lane < 16 ? 0 : n0, cols = lane < 16 ? n0 : n1;
            if (ntiles > 0) {
                const int last = n_done + ntiles - 1;
                mbar_wait(smem_u32(&bars->o_done[last & 1]), (last >> 1) & 1);
                tc_fence_after();
            }
            // DUP: warps 0 and 1 hold two parts of the same rows.  Each hands the other the columns that it finishes (of either half the
            // first or the last), and both the sums
            const int mid = DUP ? (n0 + 32) >> 6 << 5 : 0, begin = rest ? mid : 0, end = DUP && !rest ? mid : n0;
            if (DUP && warp < 2 && ntiles > 0) {
#pragma unroll 1
                for (int cc = rest ? 0 : mid; cc < (rest ? mid : n0); cc += 32) {
                    uint32_t v[32];
                    __syncwarp();
                    tmem_ld32(tlane + cc, v);
                    tmem_ld_wait();
                    if (cc < cols) {
#pragma unroll
                        for (int e = 0; e < 32; e += 4) *reinterpret_cast<uint4*>(xs + col0 + cc + e) = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
                    }
                }
                if (lane < 16) xs[LT_REST_PITCH - 4 + warp] = l;
                named_bar_sync(1, 64);
                l += xs[LT_REST_PITCH - 3 - warp];
            }
            float f = 0.f;
            float* pr = nullptr;
            if (p.nsplit > 1) {
                pr = p.partial + ((t * p.H + h) * p.nsplit + split()) * (r + 2);
                if (live && lane < 16 && !rest) { pr[r] = m * LT_LN2; pr[r + 1] = l; }
            } else if (live) {
                f = 1.f / l;
                if (p.gate != nullptr) f *= 1.f / (1.f + expf(-ldf(reinterpret_cast<const T*>(p.gate) + t * p.gate_st + h)));
            }
            T* o = reinterpret_cast<T*>(p.out) + t * p.out_st + (int64_t)h * p.out_sh + col0;
#pragma unroll 1
            for (int cc = begin; cc < end && ntiles > 0; cc += 32) {      // (a split without keys leaves its sums alone: m = -inf is not read)
                uint32_t v[32];
                __syncwarp();
                tmem_ld32(tlane + cc, v);
                tmem_ld_wait();
                if (live && cc < cols) {
                    if (DUP) {
#pragma unroll
                        for (int e = 0; e < 32; e += 4) {
                            const float4 x = *reinterpret_cast<const float4*>(xs + col0 + cc + e);
                            v[e] = __float_as_uint(__uint_as_float(v[e]) + x.x); v[e + 1] = __float_as_uint(__uint_as_float(v[e + 1]) + x.y);
                            v[e + 2] = __float_as_uint(__uint_as_float(v[e + 2]) + x.z); v[e + 3] = __float_as_uint(__uint_as_float(v[e + 3]) + x.w);
                        }
                    }
                    if (p.nsplit > 1) {
#pragma unroll
                        for (int e = 0; e < 32; e += 2)
                            *reinterpret_cast<float2*>(pr + col0 + cc + e) = make_float2(__uint_as_float(v[e]), __uint_as_float(v[e + 1]));
                    } else if (p.out_vec) {
#pragma unroll
                        for (int e = 0; e < 32; e += 8) {
                            uint32_t x[4];
#pragma unroll
                            for (int k = 0; k < 4; k++) x[k] = pack2<T>(__uint_as_float(v[e + 2 * k]) * f, __uint_as_float(v[e + 2 * k + 1]) * f);
                            *reinterpret_cast<uint4*>(o + cc + e) = make_uint4(x[0], x[1], x[2], x[3]);
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 32; e++) stf(o + cc + e, __uint_as_float(v[e]) * f);
                    }
                }
            }
            __syncwarp();
        }
        tc_fence_before();
        __syncthreads();                             // the next segment overwrites the queries; its first products overwrite O
        tc_fence_after();
        n_done += ntiles;
        if ((solo >= 0 || *tainted == pass) && ++solo < n) continue;
        solo = -1;
        i0 += n;
    }
    if (warp == LT_MMA_WARP) tmem_dealloc<512>(tmem);
}

bool latent_tc_supported(int r, int dr) { return r % 64 == 0 && r <= 512 && dr % 16 == 0 && dr <= 64; }

int launch_latent_attn_tc(LatentTc& p, bool portions, sllm_dtype_t dtype, cudaStream_t stream) {
    p.hp_log2 = 0;
    while ((1 << p.hp_log2) < p.H && p.hp_log2 < 6) p.hp_log2++;
    p.qt = portions ? LT_ROWS >> p.hp_log2 : 1;
    dim3 grid((unsigned)cdiv(p.num_tokens, p.qt), (unsigned)cdiv(p.H, 1 << p.hp_log2), (unsigned)p.nsplit);
    // SMs that are left over take segments of CTAs in whose tokens a sequence ends: their passes would come one after the other (three prompts
    // of 33 tokens, 32 heads: 38 us in 50 CTAs, 16 in 100)
    int num_sms = 0;
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, current_device());
    const int64_t share = portions ? num_sms / ((int64_t)grid.x * grid.y * grid.z) : 1;
    if (share > 1) grid.z *= (unsigned)(share > p.qt ? p.qt : share);
    const int full = p.r == 512 && p.dr == 64, rows = grid.z > (unsigned)p.nsplit ? LT_SHARED : !portions && p.hp_log2 <= 4 ? LT_SINGLES : LT_PROMPTS;
    if (portions && rows == LT_PROMPTS && latent_prompt_takes(p, grid, num_sms))
        if (const int rc = launch_latent_attn_prompt(p, grid, dtype, stream); rc >= 0) return rc;
    SLLM_DISPATCH_DTYPE(dtype, {
        static unsigned long long configured = 0;
        void (*kernels[2][3])(LatentTc) = {
            {latent_attn_tc_kernel<T, false, LT_PROMPTS>, latent_attn_tc_kernel<T, false, LT_SINGLES>, latent_attn_tc_kernel<T, false, LT_SHARED>},
            {latent_attn_tc_kernel<T, true, LT_PROMPTS>, latent_attn_tc_kernel<T, true, LT_SINGLES>, latent_attn_tc_kernel<T, true, LT_SHARED>}};
        if (first_use_on_this_device(configured)) {
            for (auto& row : kernels)
                for (auto k : row) {
                    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM);
                    SLLM_REQUIRE(e == cudaSuccess, "latent_attention: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
                }
        }
        launch_early(kernels[full][rows], grid, LT_THREADS, LT_SMEM, stream, p);
    });
    return check_launch("latent_attention (tcgen05)");
}

}  // namespace sllm
