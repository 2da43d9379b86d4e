// Window attention for prompt rows in 16-bit storage on the fifth-generation tensor cores (tcgen05 + TMEM): the same function as
// window_attn.cu, whose head comment gives the definition, the cache rows and the options.
//
// A CTA owns two tiles of 128 query ROWS of one key/value group, row = (token, head of the group) with the heads padded to a power of
// two: 64 tokens for four heads per group.  Tokens are walked in segments (runs of one sequence at consecutive positions), so any order
// of rows is correct; a segment's rows share ONE list of keys (kept first positions, then the window), taken in steps of 80.
//   warps 0, 2   producers: cache rows through the block table into a four-stage ring, in TMA boxes of 16 rows (BOXES) or by cp.async (keys past
//                the segment's last position are zero)
//   warps 1, 3   product issuers of tile A / B:  S_X(j + 1) = Q_X . K(j + 1) as soon as S_X(j) is in registers,
//                O_X += P_X(j) . V(j) when P_X(j) is there; with shared_kv the key tile is also the value tile
//   warps 4-7    queries, softmax and output of tile A, warps 8-11 of tile B: thread = query row = TMEM lane, P as 16-bit A operand in TMEM,
//                O rescaled when a row's running maximum grows (a reference that trails it by up to 2^8 is 4 % faster, but the
//                largest weight is then not 1 and takes a rounding as well: 2.38e-3 instead of 2.33e-3 off 64 bits in bf16)
// TMEM: S_A 0..79, S_B 80..159, P_A 160..199, P_B 200..239, O_A 256..383, O_B 384..511 (the layout of the prefill kernel: 80 keys are the
// most that leave scores and P places of their own).
// A weight of exactly 0 times a value that is not finite is NaN, so a key that one row of a pass sees and another does not may reach both.
// Where a row's sum of weights is finite but its O is not, and such a value is found among the keys that only some tokens of the segment
// see, the segment is done over, token by token, with the keys that the token does not see left zero: a result depends on its own keys only.
//
// Measured on B200, bf16, 16 heads on 4 key/value heads of 128 entries, window 1024: prompts of 2048, 242 and 1507 tokens beside forty decoded
// ones 312 us with the mma.sync kernel of window_attn.cu for the prompts -> 118 us, 91 with the decoded rows beside the prompts' last CTAs, 83 with
// boxes (the prompts alone 85 -> 74, one of 2048 51 -> 42, 600 rows at 1500 41 -> 31, 32 heads at 1000, window 2048 170 -> 144; with the long
// CTAs of all groups first 74 -> 64, 144 -> 117).  Two rounds of CTAs here; a CTA's step of 80 keys is 2000 cycles of softmax, its queries 10 k, its
// output 10 k (gates one by one 15 k).
//
// EXT: the kernel knows slopes, kept first positions, gates per head, shared_kv rows and learned sinks; CAP: a tanh cap on the scores;
// FULL: heads of 128 + 128 entries without turned ones beside shared keys (the producers are bound by their instructions).
#include "mma_helpers.cuh"
#include "tc_helpers.cuh"
#include "typed_io.cuh"
#include "window_attn_tc.cuh"

namespace sllm {

using namespace tc;

constexpr int WX_ROWS = 128, WX_BK = 80, WX_STAGES = 4, WX_THREADS = 384;
constexpr int WX_QCHUNK = WX_ROWS * 128;              // 128 rows x 64 columns
constexpr int WX_CHUNK = WX_BK * 128;                 // 80 keys x 64 columns
constexpr int WX_CHUNKS = 4;                          // 64-column chunks of a stage: keys, then values (shared_kv: keys only)
constexpr int WX_STAGE = WX_CHUNKS * WX_CHUNK;
constexpr int WX_Q_BYTES = 2 * WX_QCHUNK;
constexpr int WX_INV_OFF = 2 * WX_Q_BYTES + WX_STAGES * WX_STAGE;                 // [stage][80] fp32: the keys' 1 / rms
constexpr int WX_MISC_OFF = WX_INV_OFF + WX_STAGES * WX_BK * 4;
constexpr int WX_SMEM = WX_MISC_OFF + 256;
constexpr int WX_S_COL = 0, WX_P_COL = 160, WX_O_COL = 256;      // tile B: + 80, + 40, + 128
constexpr float WX_LOG2E = 1.4426950408889634f;
// registers: 384 threads are launched with 168 each; the softmax warpgroups hold a row of scores and of P
constexpr int WX_REGS_FEW = 88, WX_REGS_MANY = 208;
static_assert(WX_REGS_FEW + 2 * WX_REGS_MANY <= 3 * 168, "the warpgroups' shares must fit what the block was launched with");
constexpr int WX_LAG = 1;                             // steps whose rows are in flight behind the one being asked for

struct WindowTcBars {
    uint64_t full[WX_STAGES], empty[WX_STAGES];
    uint64_t s_full[2], s_empty[2], p_full[2], p_empty[2];
    uint64_t landed[2];                              // [keys, values]: boxes of a step whose unseen rows have yet to become zero
};

// y / (1 + e^-z), two at a time: the quick reciprocal and one step of Newton's iteration, r + r (1 - d r), which leaves about half a unit in the last place
// and has no branch, so that the gates of a row are worked on together (with a quotient rounded exactly the case below took 127 us
// instead of 115).  Five to six instructions a gate: a row's 128 take 1.9 k cycles of its warp when it has the scheduler to itself (one by one 3.8 k).
__device__ __forceinline__ float rcp_quick(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 gate_pair(float2 y, float2 z) {
    const float2 one = make_float2(1.f, 1.f), t = mul2(z, make_float2(-WX_LOG2E, -WX_LOG2E));
    const float2 d = add2(make_float2(fast_exp2_tc(t.x), fast_exp2_tc(t.y)), one), r = make_float2(rcp_quick(d.x), rcp_quick(d.y));
    const float2 low = make_float2(-fminf(d.x, 0x1p127f), -fminf(d.y, 0x1p127f));      // r is 0 from d = 2^126 on
    return mul2(y, fma2(r, fma2(low, r, one), r));
}

// BOXES: keys and values come in TMA boxes of 16 cache rows, each producer warp its half of a step's columns (a step's 5120 16-byte pieces by cp.async take
// two warps 2500 to 3000 cycles to ask for, softmax and products 2100)
template <typename T, bool EXT, bool CAP, bool FULL, bool BOXES>
__global__ void __launch_bounds__(WX_THREADS, 1) window_attn_tc_kernel(const __grid_constant__ CUtensorMap map, const WindowTc p) {
    static_assert(!BOXES || (FULL && !EXT), "boxes of 128 + 128 columns, of one run of positions");
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* q_sm = smem;                             // [tile][chunk][128 rows][128 B]
    uint8_t* kv_sm = smem + 2 * WX_Q_BYTES;           // [stage][chunk][80 keys][128 B]
    float* inv_sm = reinterpret_cast<float*>(smem + WX_INV_OFF);
    WindowTcBars* bars = reinterpret_cast<WindowTcBars*>(smem + WX_MISC_OFF);
    uint32_t* tmem_s = reinterpret_cast<uint32_t*>(smem + WX_MISC_OFF + sizeof(WindowTcBars));
    volatile int* tainted = reinterpret_cast<int*>(tmem_s + 1);      // [2]: the last pass in which O was not finite; ... that is done over
    static_assert(sizeof(WindowTcBars) + 12 <= 256, "");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool shared_kv = EXT && p.shared_kv;
    const int krot = EXT && !FULL ? p.krot : 0, keep_first = EXT ? p.keep_first : 0;
    const int dk = FULL ? 128 : p.dk, dv = FULL ? 128 : p.dv, KW = dk + krot, hq = p.H / p.G, hqp = 1 << p.hqp_log2;
    const int kch = (KW + 63) >> 6, vch = shared_kv ? 0 : (dv + 63) >> 6;         // chunks of a key / value row
    // The last tokens of a prompt have the most keys: first, in all groups (p.group_blocks: in one group behind the other)
    const int behind = gridDim.x - 1 - blockIdx.x, of = p.group_blocks ? p.group_blocks : p.G, k = behind / of;
    const int block = p.group_blocks ? behind - k * of : k, g = p.group_blocks ? k : behind - k * of;
    const int t_first = block * p.qt;
    const int ntok = min(p.qt, p.num_rows - t_first);

    if (tid == 0) {
        tainted[0] = tainted[1] = 0;
        for (int s = 0; s < WX_STAGES; s++) { mbar_init(smem_u32(&bars->full[s]), 2); mbar_init(smem_u32(&bars->empty[s]), 2); }
        for (int x = 0; x < 2; x++) {
            mbar_init(smem_u32(&bars->s_full[x]), 1); mbar_init(smem_u32(&bars->s_empty[x]), 128);
            mbar_init(smem_u32(&bars->p_full[x]), 128); mbar_init(smem_u32(&bars->p_empty[x]), 1);
            mbar_init(smem_u32(&bars->landed[x]), 1);
        }
        mbar_fence_init();
        if constexpr (BOXES) tma_prefetch_desc(&map);
    }
    if (warp == 1) tmem_alloc<512>(smem_u32(tmem_s));
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_s;
    wait_previous();
    launch_next();

    // ---- a segment: tokens ts .. ts + n - 1 of one sequence at positions pos0 ..
    struct Segment { int ts, n, seq, pos0, lo, hi, nk, steps_a, steps_b, end_a, end_b; };
    const int tpt = WX_ROWS >> p.hqp_log2;                                        // tokens per tile
    const int vkeep = EXT && p.window > 0 ? keep_first : 0;                        // list entries below it are kept positions
    auto first_seen = [&](int pos) {                  // first position of the window (and chunk) of a query at `pos`
        int a = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
        if (p.chunk > 0) a = max(a, pos / p.chunk * p.chunk);
        return a;
    };
    auto segment = [&](int i0) {
        Segment s;
        s.ts = t_first + i0;
        const int left = ntok - i0;
        s.seq = p.tok_seq[s.ts]; s.pos0 = p.tok_pos[s.ts];
        s.n = left;
        for (int b = 0; b < left; b += 64) {              // (all loads of 64 tokens in flight together)
            const int i = min(b + lane, left - 1), k = min(i + 32, left - 1);
            const int qi = p.tok_seq[s.ts + i], qk = p.tok_seq[s.ts + k], pi = p.tok_pos[s.ts + i], pk = p.tok_pos[s.ts + k];
            const uint32_t cut = __ballot_sync(0xffffffffu, qi != s.seq || pi != s.pos0 + i), later = __ballot_sync(0xffffffffu, qk != s.seq || pk != s.pos0 + k);
            if (cut) { s.n = b + __ffs(cut) - 1; break; }
            if (later) { s.n = b + 31 + __ffs(later); break; }
        }
        s.lo = first_seen(s.pos0); s.hi = s.pos0 + s.n - 1;
        if constexpr (BOXES) s.lo &= ~15;                 // (a box's first row)
        s.nk = EXT && p.window > 0 ? min(keep_first, s.lo) : 0;
        const int na = min(s.n, tpt), nb = s.n - na;
        // entry v of the list of keys is position v (v < nk) or v - nk + lo; entries a tile's last token sees
        s.end_a = s.nk + s.pos0 + na - s.lo; s.end_b = nb > 0 ? s.nk + s.hi - s.lo + 1 : 0;
        s.steps_a = (s.end_a + WX_BK - 1) / WX_BK; s.steps_b = (s.end_b + WX_BK - 1) / WX_BK;
        return s;
    };
    // steps of the passes before (of the ring, of each tile): the barriers' phases follow from them
    int n_done = 0, done_a = 0, done_b = 0;
    int pass = 0, solo = -1;                          // solo >= 0: the pass is for this token of the segment alone
    const int kofs = p.koff + g * KW, vofs = p.G * dk + (g / p.vshare) * dv;       // the group's keys and values in a cache row
    auto row_of = [&](const int* bt, int nk, int lo, int v) {      // cache row of list entry v
        const int kp = v < nk ? v : v - nk + lo;
        const int b = kp / p.block_size;
        return ((long long)bt[b] * p.n_slots + p.slot) * p.block_size + (kp - b * p.block_size);
    };
    // what a pass ends with: true if the segment is taken once more (its end was a barrier)
    auto again = [&](const Segment& s, bool search) {
        if (solo < 0) {
            if (tainted[0] != pass) return false;
            if (search) {
                const int all_lo = s.nk + first_seen(s.hi) - s.lo, all_hi = s.nk + s.pos0 - s.lo, total = max(s.end_a, s.end_b);
                const int* bt = p.block_table + (int64_t)s.seq * p.max_blocks_per_seq;
                const T* values = reinterpret_cast<const T*>(p.cache) + (shared_kv ? kofs : vofs);
                for (int v = vkeep + warp - 4; v < total; v += WX_THREADS / 32 - 4) {
                    if (v >= all_lo && v <= all_hi) continue;
                    const T* row = values + row_of(bt, s.nk, s.lo, v) * p.row_elems;
                    bool odd = false;
                    for (int d = lane; d < dv; d += 32) { const float x = ldf(row + d); odd |= x - x != 0.f; }
                    if (odd) tainted[1] = pass;
                }
            }
            __syncthreads();
            if (tainted[1] != pass) return false;
        }
        if (++solo < s.n) return true;
        solo = -1;
        return false;
    };
    if (warp < 4) {
        reg_dec<WX_REGS_FEW>();
        int landed_done = 0;                          // phases of `landed`
        for (int i0 = 0; i0 < ntok;) {
            pass++;
            const Segment sg = segment(i0);
            const int n = sg.n, lo = sg.lo, nk = sg.nk, nsteps = max(sg.steps_a, sg.steps_b);
            // list entries that are visible: all of them, or those of one token
            const int* bt = p.block_table + (int64_t)sg.seq * p.max_blocks_per_seq;
            const int own = sg.pos0 + max(solo, 0), total = solo < 0 ? max(sg.end_a, sg.end_b) : nk + own - lo + 1;
            const int hidden = solo < 0 ? 0 : nk + first_seen(own) - lo;             // entries vkeep .. hidden - 1 are not
            if (BOXES && (warp == 0 || warp == 2)) {
                // ======================================================= producers: warp 0 the keys, warp 2 the values; lanes 0 .. 4 a box each
                const int seen = (solo < 0 ? first_seen(sg.pos0) : first_seen(own)) - lo;      // entries seen .. total - 1 are visible
                const int col = warp == 0 ? kofs : vofs;
                auto box_row = [&](int j) {
                    const int kp = lo + j * WX_BK + 16 * lane;
                    if (lane >= WX_BK / 16 || j >= nsteps || kp >= lo + total) return -1;
                    const int b = kp / p.block_size;
                    return (int)(((long long)bt[b] * p.n_slots + p.slot) * p.block_size + (kp - b * p.block_size));
                };
                int next = box_row(0);
                for (int j = 0; j < nsteps; j++) {
                    const int it = n_done + j, st = it % WX_STAGES, row = next;
                    next = box_row(j + 1);
                    const bool ragged = j * WX_BK < seen || (j + 1) * WX_BK > total;
                    const uint32_t full = smem_u32(&bars->full[st]), bar = ragged ? smem_u32(&bars->landed[warp >> 1]) : full;
                    uint8_t* half = kv_sm + st * WX_STAGE + warp * WX_CHUNK;                  // this warp's two chunks
                    const int boxes = __popc(__ballot_sync(0xffffffffu, row >= 0));
                    if (lane == 0) {
                        mbar_wait(smem_u32(&bars->empty[st]), ((it / WX_STAGES) & 1) ^ 1);
                        mbar_arrive_expect_tx(bar, (uint32_t)boxes * 16 * 256);
                    }
                    __syncwarp();
                    if (row >= 0) {
                        tma_load_2d(smem_u32(half) + lane * 2048, &map, bar, col, row);
                        tma_load_2d(smem_u32(half) + WX_CHUNK + lane * 2048, &map, bar, col + 64, row);
                    }
                    if (!ragged) continue;
                    mbar_wait(bar, landed_done++ & 1);        // rows that are not seen become zero
                    for (int r = lane >> 4; r < WX_BK; r += 2)
                        if (j * WX_BK + r < seen || j * WX_BK + r >= total)
                            *reinterpret_cast<uint4*>(half + ((lane >> 3) & 1) * WX_CHUNK + r * 128 + (lane & 7) * 16) = make_uint4(0, 0, 0, 0);
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(full);
                }
            } else if (warp == 0 || warp == 2) {
                // ======================================================= producers: keys 40 (warp / 2) .. of every step, eight lanes a 128-byte piece
                const int r0 = 20 * warp, piece = lane & 7;
                const T* cache = reinterpret_cast<const T*>(p.cache);
                auto key_row = [&](int v) { return v >= total || (v < hidden && v >= vkeep) ? -1ll : row_of(bt, nk, lo, v); };      // -1: not visible
                auto signal = [&](int j) {
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&bars->full[(n_done + j) % WX_STAGES]));
                };
                long long ra = key_row(r0 + lane), rb = lane < 8 ? key_row(r0 + 32 + lane) : -1ll;
                for (int j = 0; j < nsteps; j++) {
                    const long long a = ra, b = rb;
                    if (j + 1 < nsteps) {
                        ra = key_row((j + 1) * WX_BK + r0 + lane);
                        rb = lane < 8 ? key_row((j + 1) * WX_BK + r0 + 32 + lane) : -1ll;
                    }
                    const int it = n_done + j, st = it % WX_STAGES;
                    mbar_wait(smem_u32(&bars->empty[st]), ((it / WX_STAGES) & 1) ^ 1);
                    const uint32_t stage = smem_u32(kv_sm + st * WX_STAGE);
#pragma unroll 2
                    for (int i = 0; i < 10; i++) {
                        const int l = 4 * i + (lane >> 3), row = r0 + l;
                        const long long ri = __shfl_sync(0xffffffffu, i < 8 ? a : b, l & 31);
                        const int bytes = ri >= 0 ? 16 : 0;
                        const T* src = ri >= 0 ? cache + ri * p.row_elems : cache;
                        const uint32_t dst = stage + swizzled(row, piece);
                        if constexpr (FULL) {             // (a row that is not there reads nothing, wherever src points)
                            const T* ks = src + kofs + piece * 8;
                            cp_async16(dst, ks, bytes); cp_async16(dst + WX_CHUNK, ks + 64, bytes);
                            if (!shared_kv) {
                                const T* vs = src + vofs + piece * 8;
                                cp_async16(dst + 2 * WX_CHUNK, vs, bytes); cp_async16(dst + 3 * WX_CHUNK, vs + 64, bytes);
                            }
                        } else {
                            for (int c = 0; c < kch; c++)
                                if (c * 64 + piece * 8 < KW) cp_async16(dst + c * WX_CHUNK, bytes ? src + kofs + c * 64 + piece * 8 : src, bytes);
                            for (int c = 0; c < vch; c++)
                                if (c * 64 + piece * 8 < dv)
                                    cp_async16(dst + (kch + c) * WX_CHUNK, bytes ? src + vofs + c * 64 + piece * 8 : src, bytes);
                        }
                        if (EXT && shared_kv && piece == 0) {
                            float* to = inv_sm + st * WX_BK + row;
                            if (bytes) cp_async4(smem_u32(to), src + 2 * g);
                            else *to = 0.f;
                        }
                    }
                    cp_async_commit();
                    if (j >= WX_LAG) { cp_async_wait<WX_LAG>(); signal(j - WX_LAG); }
                }
                cp_async_wait<0>();
                for (int j = max(0, nsteps - WX_LAG); j < nsteps; j++) signal(j);
            } else {
                // ======================================================= product issuers (the warp stays converged, one elected lane issues)
                const int x = warp >> 1;
                const int mine = x == 0 ? sg.steps_a : sg.steps_b, end = x == 0 ? sg.end_a : sg.end_b, x_done = x == 0 ? done_a : done_b;
                const uint32_t idesc_s = make_instr_desc(WX_ROWS, WX_BK, UmmaFmt<T>::value, 0, 0);
                const uint32_t idesc_o = make_instr_desc(WX_ROWS, dv, UmmaFmt<T>::value, 0, 1);
                const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
                const uint32_t s_addr = tm + WX_S_COL + x * WX_BK, p_addr = tm + WX_P_COL + x * (WX_BK / 2), o_addr = tm + WX_O_COL + x * 128;
                const uint64_t dq = make_smem_desc(smem_u32(q_sm + x * WX_Q_BYTES), 16, 1024);
                const uint64_t dk0 = make_smem_desc(smem_u32(kv_sm), 16, 1024), dv0 = make_smem_desc(smem_u32(kv_sm), WX_CHUNK, 1024);
                const uint32_t vfirst = (uint32_t)((vch > 0 ? kch : 0) * WX_CHUNK) >> 4;
                const int kd_steps = dk >> 4;
                auto scores = [&](int j) {
                    const int it = n_done + j, st = it % WX_STAGES;
                    const uint64_t kd = dk0 + (uint64_t)((st * WX_STAGE) >> 4);
                    mbar_wait(smem_u32(&bars->full[st]), (it / WX_STAGES) & 1);
                    if (j > 0) mbar_wait(smem_u32(&bars->s_empty[x]), (x_done + j - 1) & 1);
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            if (k < kd_steps) {
                                const int col = krot + 16 * k;
                                umma_ss(s_addr, dq + (uint64_t)(((k >> 2) * WX_QCHUNK + (k & 3) * 32) >> 4),
                                        kd + (uint64_t)(((col >> 6) * WX_CHUNK + (col & 63) * 2) >> 4), idesc_s, k > 0);
                            }
                        umma_commit(smem_u32(&bars->s_full[x]));
                    }
                    __syncwarp();
                };
                named_bar_sync(1, WX_THREADS - 64);       // the queries are staged
                if (mine > 0) {
                    scores(0);
                    for (int j = 0; j < mine; j++) {
                        const int xi = x_done + j;
                        if (j + 1 < mine) scores(j + 1);
                        const int st = (n_done + j) % WX_STAGES;
                        const int k16 = min(WX_BK / 16, (end - j * WX_BK + 15) / 16);         // none past the last key the tile can see
                        const uint64_t vd = dv0 + (uint64_t)((st * WX_STAGE) >> 4) + vfirst;
                        mbar_wait(smem_u32(&bars->p_full[x]), xi & 1);
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int k = 0; k < WX_BK / 16; k++)
                                if (k < k16) umma_ts(o_addr, p_addr + 8 * k, vd + (uint64_t)((k * 2048) >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
                            umma_commit(smem_u32(&bars->empty[st]));
                            umma_commit(smem_u32(&bars->p_empty[x]));
                        }
                        __syncwarp();
                    }
                    // the last scores' s_empty is waited for by nobody: its phase is taken by the count x_done
                }
                // steps that only the other tile takes: hand the stages on once they have been filled (never a phase ahead)
                for (int j = mine; j < nsteps; j++) {
                    const int it = n_done + j, st = it % WX_STAGES;
                    mbar_wait(smem_u32(&bars->full[st]), (it / WX_STAGES) & 1);
                    if (lane == 0) mbar_arrive(smem_u32(&bars->empty[st]));
                }
            }
            tc_fence_before();
            __syncthreads();                          // the next segment overwrites the queries; its first products overwrite O
            tc_fence_after();
            n_done += nsteps; done_a += sg.steps_a; done_b += sg.steps_b;
            if (!again(sg, false)) i0 += n;
        }
    } else {
        reg_inc<WX_REGS_MANY>();
        const int x = (warp - 4) >> 2, quad = warp & 3, row = quad * 32 + lane;
        for (int i0 = 0; i0 < ntok;) {
            pass++;
            const Segment sg = segment(i0);
            const int ts = sg.ts, n = sg.n, pos0 = sg.pos0, lo = sg.lo, nk = sg.nk, nsteps = max(sg.steps_a, sg.steps_b);
            // ---- queries of both tiles, half a warp per row, eight entries a lane: (norm,) rotation, (norm) in fp32, rounded to the storage type
            {
                const int me = warp - 4;
                const int l16 = lane & 15, d = l16 * 8, half = p.rot_dims >> 1;
                const int nrows = n > tpt ? 2 * WX_ROWS : WX_ROWS;
                auto sum16 = [&](float v) {
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    return v;
                };
                auto stage_row = [&](int row, const float (&x)[8]) {
                    if (d < dk) {
                        const uint4 v = make_uint4(pack2<T>(x[0], x[1]), pack2<T>(x[2], x[3]), pack2<T>(x[4], x[5]), pack2<T>(x[6], x[7]));
                        *reinterpret_cast<uint4*>(q_sm + (row >> 7) * WX_Q_BYTES + (d >> 6) * WX_QCHUNK + swizzled(row & 127, (d & 63) >> 3)) = v;
                    }
                };
                if (p.q_fast) {
                    // neighbouring pairs turn, 16-byte loads: four rows' loads are in flight before the first is used
                    const int dc = min(d, dk - 8), dr = min(d, p.rot_dims - 8) >> 1;
                    float nw[8];
#pragma unroll
                    for (int e = 0; e < 8; e++) nw[e] = p.qnorm_w != nullptr ? p.qnorm_w[dc + e] : 1.f;
                    const bool turns = d < p.rot_dims;
                    // 64 rows on, a lane's row is that of the same head (at most 64 of a group) some tokens on: its pointers move by constants
                    const int start = 2 * me + (lane >> 4), hop = 64 >> p.hqp_log2;
                    const T* qp[4];
                    const float* cp[4];
                    const float* sp[4];
#pragma unroll
                    for (int b = 0; b < 4; b++) {
                        const int row = start + 16 * b;
                        const int64_t t = ts + (row >> p.hqp_log2);
                        qp[b] = reinterpret_cast<const T*>(p.q) + t * p.q_st + (int64_t)(g * hq + min(row & (hqp - 1), hq - 1)) * dk + dc;
                        cp[b] = p.cosb + t * half + dr; sp[b] = p.sinb + t * half + dr;
                    }
                    const int64_t q_hop = hop * p.q_st;
                    const int a_hop = hop * half;
                    // The next rows are on their way while these are turned; not in EXT kernels, whose registers they cost more than their latency (us, ahead /
                    // not, shared keys, 32 / 8 heads: two of up to 100 tokens 33.6 / 32.5, 16 of up to 128 47.1 / 45.2, three of up to 2048 105 / 104)
                    constexpr bool AHEAD = !EXT;
                    Vec8<T> nu[4];
                    float4 nc[4], ns[4];
#pragma unroll
                    for (int b = 0; b < 4; b++) nc[b] = ns[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                    auto ask = [&](int r0) {
#pragma unroll
                        for (int b = 0; b < 4; b++) {
                            if (((r0 + 16 * b) >> p.hqp_log2) < n) {          // (other rows are made zero below)
                                nu[b] = ld_vec8(qp[b]);
                                if (p.rot_dims > 0) { nc[b] = *reinterpret_cast<const float4*>(cp[b]); ns[b] = *reinterpret_cast<const float4*>(sp[b]); }
                            }
                            qp[b] += q_hop; cp[b] += a_hop; sp[b] += a_hop;
                        }
                    };
                    if (AHEAD) ask(start);
#pragma unroll 1
                    for (int r0 = start; r0 < nrows; r0 += 64) {
                        if (!AHEAD) ask(r0);
                        Vec8<T> u[4];
                        float4 c4[4], s4[4];
#pragma unroll
                        for (int b = 0; b < 4; b++) { u[b] = nu[b]; c4[b] = nc[b]; s4[b] = ns[b]; }
                        if (AHEAD && r0 + 64 < nrows) ask(r0 + 64);
#pragma unroll
                        for (int b = 0; b < 4; b++) {
                            const int row = r0 + 16 * b;
                            const bool live = (row >> p.hqp_log2) < n && (row & (hqp - 1)) < hq && d < dk;
                            float x[8];
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const float2 f = Traits<T>::to_f2(u[b].v[e]);
                                x[2 * e] = live ? f.x : 0.f; x[2 * e + 1] = live ? f.y : 0.f;
                            }
                            if (p.qnorm_w != nullptr) {
                                float ss = 0.f;
#pragma unroll
                                for (int e = 0; e < 8; e++) ss += x[e] * x[e];
                                const float inv = 1.f / sqrtf(sum16(ss) / (float)dk + p.prenorm_eps);
#pragma unroll
                                for (int e = 0; e < 8; e++) x[e] *= inv * nw[e];
                            }
                            if (turns) {
                                const float cs[4] = {c4[b].x, c4[b].y, c4[b].z, c4[b].w}, sn[4] = {s4[b].x, s4[b].y, s4[b].z, s4[b].w};
#pragma unroll
                                for (int e = 0; e < 4; e++) {
                                    const float v = x[2 * e], w = x[2 * e + 1];
                                    x[2 * e] = v * cs[e] - w * sn[e]; x[2 * e + 1] = w * cs[e] + v * sn[e];
                                }
                            }
                            if (p.qk_norm_eps >= 0.f) {
                                float ss = 0.f;
#pragma unroll
                                for (int e = 0; e < 8; e++) ss += x[e] * x[e];
                                const float inv = 1.f / sqrtf(sum16(ss) / (float)dk + p.qk_norm_eps);
#pragma unroll
                                for (int e = 0; e < 8; e++) x[e] *= inv;
                            }
                            if (row < nrows) stage_row(row, x);
                        }
                    }
                } else
#pragma unroll 1
                for (int r0 = 2 * me; r0 < nrows; r0 += 16) {
                    const int row = r0 + (lane >> 4), tr = row >> p.hqp_log2, hh = row & (hqp - 1);
                    const bool live = tr < n && hh < hq && d < dk;
                    const int64_t t = ts + tr;
                    const T* qr = reinterpret_cast<const T*>(p.q) + t * p.q_st + (int64_t)(g * hq + hh) * dk;
                    float x[8], y[8];                     // the lane's entries; with `halves` the partners of those that turn
                    const bool turns = live && d < p.rot_dims;
                    const int dp = d < half ? d + half : d - half;                    // partner group (halves)
#pragma unroll
                    for (int e = 0; e < 8; e++) { x[e] = 0.f; y[e] = 0.f; }
                    if (live) {
                        if (p.q_vec) {
                            const Vec8<T> u = ld_vec8(qr + d);
#pragma unroll
                            for (int e = 0; e < 4; e++) { const float2 f = Traits<T>::to_f2(u.v[e]); x[2 * e] = f.x; x[2 * e + 1] = f.y; }
                            if (p.halves && turns) {
                                const Vec8<T> w = ld_vec8(qr + dp);
#pragma unroll
                                for (int e = 0; e < 4; e++) { const float2 f = Traits<T>::to_f2(w.v[e]); y[2 * e] = f.x; y[2 * e + 1] = f.y; }
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; e++) x[e] = ldf(qr + d + e);
                            if (p.halves && turns) {
#pragma unroll
                                for (int e = 0; e < 8; e++) {
                                    const int j = d + e;
                                    y[e] = j < p.rot_dims ? ldf(qr + (j < half ? j + half : j - half)) : 0.f;
                                }
                            }
                        }
                    }
                    if (p.qnorm_w != nullptr) {
                        float ss = 0.f;
#pragma unroll
                        for (int e = 0; e < 8; e++) ss += x[e] * x[e];
                        const float inv = 1.f / sqrtf(sum16(ss) / (float)dk + p.prenorm_eps);
                        if (live) {
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                x[e] *= inv * p.qnorm_w[d + e];
                                const int j = d + e;
                                if (p.halves && j < p.rot_dims) y[e] *= inv * p.qnorm_w[j < half ? j + half : j - half];
                            }
                        }
                    }
                    if (turns) {
                        const float* cs = p.cosb + t * half;
                        const float* sn = p.sinb + t * half;
                        if (p.halves) {
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const int j = d + e;
                                if (j < half) x[e] = x[e] * cs[j] - y[e] * sn[j];
                                else if (j < p.rot_dims) x[e] = x[e] * cs[j - half] + y[e] * sn[j - half];
                            }
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                const int i = (d >> 1) + e;
                                if (i < half) {
                                    const float a = x[2 * e], b = x[2 * e + 1];
                                    x[2 * e] = a * cs[i] - b * sn[i]; x[2 * e + 1] = b * cs[i] + a * sn[i];
                                }
                            }
                        }
                    }
                    if (p.qk_norm_eps >= 0.f) {
                        float ss = 0.f;
#pragma unroll
                        for (int e = 0; e < 8; e++) ss += x[e] * x[e];
                        const float inv = 1.f / sqrtf(sum16(ss) / (float)dk + p.qk_norm_eps);
#pragma unroll
                        for (int e = 0; e < 8; e++) x[e] *= inv;
                    }
                    stage_row(row, x);
                }
                fence_proxy_async();
                named_bar_sync(1, WX_THREADS - 64);
            }
            // ======================================================= softmax: tile x, thread = row
            const int mine = x == 0 ? sg.steps_a : sg.steps_b, x_done = x == 0 ? done_a : done_b;
            const int tr = x * tpt + (row >> p.hqp_log2), hh = row & (hqp - 1), h = g * hq + hh;
            const bool live = tr < n && hh < hq;
            const int pos = pos0 + tr;
            // visible list entries: vmin .. vmax, and those below vkeep
            const int vmax = nk + pos - lo, vmin = nk + first_seen(pos) - lo;
            // entries every live row of the tile sees without a look
            const int tr0 = x * tpt, tr1 = min(n, (x + 1) * tpt) - 1;
            const int all_lo = nk + first_seen(pos0 + tr1) - lo, all_hi = nk + pos0 + tr0 - lo;
            const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16);
            const uint32_t s_addr = tl + WX_S_COL + x * WX_BK, p_addr = tl + WX_P_COL + x * (WX_BK / 2), o_addr = tl + WX_O_COL + x * 128;
            const float c = p.scale * WX_LOG2E, cap_in = CAP ? p.scale / p.softcap : 0.f, cap_out = CAP ? p.softcap * WX_LOG2E : 0.f;
            const float slope = EXT && p.slopes != nullptr && live ? p.slopes[h] * WX_LOG2E : 0.f;
            float m_ref = p.sink > 0.f ? 0.f : -INFINITY, l = p.sink;
            if (EXT && p.sinks != nullptr && live) { m_ref = p.sinks[h] * WX_LOG2E; l = 1.f; }
            for (int j = 0; j < mine; j++) {
                const int xi = x_done + j;
                mbar_wait(smem_u32(&bars->s_full[x]), xi & 1);
                tc_fence_after();
                uint32_t r[WX_BK];
                tmem_ld32(s_addr, reinterpret_cast<uint32_t(&)[32]>(r[0]));
                tmem_ld32(s_addr + 32, reinterpret_cast<uint32_t(&)[32]>(r[32]));
                tmem_ld<16>(s_addr + 64, reinterpret_cast<uint32_t(&)[16]>(r[64]));
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->s_empty[x]));
                const int v0 = j * WX_BK;
                if constexpr (CAP || EXT) {           // scores in base 2, all factors applied
                    if (EXT && shared_kv) {
                        const int it = n_done + j;
                        mbar_wait(smem_u32(&bars->full[it % WX_STAGES]), (it / WX_STAGES) & 1);      // long there: orders the producers' writes
                        const float* iv = inv_sm + it % WX_STAGES * WX_BK;
#pragma unroll
                        for (int i = 0; i < WX_BK; i += 4) {
                            const float4 f = *reinterpret_cast<const float4*>(iv + i);
                            r[i] = __float_as_uint(__uint_as_float(r[i]) * f.x); r[i + 1] = __float_as_uint(__uint_as_float(r[i + 1]) * f.y);
                            r[i + 2] = __float_as_uint(__uint_as_float(r[i + 2]) * f.z); r[i + 3] = __float_as_uint(__uint_as_float(r[i + 3]) * f.w);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < WX_BK; i++) {
                        const float s = __uint_as_float(r[i]);
                        r[i] = __float_as_uint(CAP ? cap_out * tanhf(s * cap_in) : s * c);
                    }
                    if (EXT && p.slopes != nullptr) {
                        const float far = (float)(pos - lo + nk - v0), near = (float)(pos - v0);      // distance of entry v0 (kept: near)
#pragma unroll
                        for (int i = 0; i < WX_BK; i++)
                            r[i] = __float_as_uint(__uint_as_float(r[i]) - slope * ((v0 + i < nk ? near : far) - (float)i));
                    }
                }
                if (v0 + WX_BK - 1 > all_hi || v0 < all_lo) {
                    const int top = vmax - v0, bottom = vmin - v0, kept = vkeep - v0;
#pragma unroll
                    for (int i = 0; i < WX_BK; i++) r[i] = i <= top && (i >= bottom || (EXT && i < kept)) ? r[i] : 0xff800000u;
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int i = 0; i < WX_BK; i += 8)
#pragma unroll
                    for (int e = 0; e < 4; e++) mx[e] = max3(mx[e], __uint_as_float(r[i + 2 * e]), __uint_as_float(r[i + 2 * e + 1]));
                const float cc = CAP || EXT ? 1.f : c;
                const float m_new = fmaxf(m_ref, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * cc);
                const bool need = m_new > m_ref;
                const float alpha = need ? fast_exp2_tc(m_ref - m_new) : 1.f;
                l *= alpha;
                if (j > 0 && __any_sync(0xffffffffu, need)) {
                    mbar_wait(smem_u32(&bars->p_empty[x]), (xi - 1) & 1);          // the products of step j - 1 are done: O is stable
                    tc_fence_after();
                    if constexpr (FULL && !EXT) {     // a round trip to TMEM takes as long for 64 columns as for 16
#pragma unroll 1
                        for (int d = 0; d < 128; d += 64) {
                            uint32_t t[2][32];
                            tmem_ld32(o_addr + d, t[0]);
                            tmem_ld32(o_addr + d + 32, t[1]);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 64; i += 2) {
                                const float2 y = mul2(make_float2(__uint_as_float(t[i >> 5][i & 31]), __uint_as_float(t[i >> 5][(i & 31) + 1])), make_float2(alpha, alpha));
                                t[i >> 5][i & 31] = __float_as_uint(y.x); t[i >> 5][(i & 31) + 1] = __float_as_uint(y.y);
                            }
                            tmem_st32(o_addr + d, t[0]);
                            tmem_st32(o_addr + d + 32, t[1]);
                        }
                    } else {
#pragma unroll 1
                        for (int d = 0; d < dv; d += 16) {
                            uint32_t t[16];
                            tmem_ld<16>(o_addr + d, t);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; i++) t[i] = __float_as_uint(__uint_as_float(t[i]) * alpha);
                            tmem_st16(o_addr + d, t);
                        }
                    }
                }
                if (need) m_ref = m_new;
                const float sub = m_ref == -INFINITY ? 0.f : -m_ref;              // nothing seen yet
                // the sum takes the rounded weights (of the exact ones: 2.332e-3 instead of 2.319e-3 off 64 bits in bf16; the mma.sync kernel with
                // its steps of 32 keys, whose maxima leave more weights exact, 2.321e-3)
                float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                const float2 neg_m = make_float2(sub, sub), c2 = make_float2(cc, cc);
                uint32_t w[WX_BK / 2];
#pragma unroll
                for (int i = 0; i < WX_BK / 2; i++) {
                    const float2 e = fma2(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), c2, neg_m);
                    w[i] = pack2<T>(fast_exp2_tc(e.x), fast_exp2_tc(e.y));
                    ls[i & 1] = add2(ls[i & 1], Traits<T>::to_f2(*reinterpret_cast<typename Traits<T>::T2*>(&w[i])));
                }
                if (j > 0) { mbar_wait(smem_u32(&bars->p_empty[x]), (xi - 1) & 1); tc_fence_after(); }      // P of step j - 1 has been read
                tmem_st32(p_addr, reinterpret_cast<uint32_t(&)[32]>(w[0]));
                tmem_st8(p_addr + 32, reinterpret_cast<uint32_t(&)[8]>(w[32]));
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(smem_u32(&bars->p_full[x]));
                l += (ls[0].x + ls[0].y) + (ls[1].x + ls[1].y);
            }
            if (mine > 0) {
                // ---- output row: normalise, (turn back,) gate, store
                mbar_wait(smem_u32(&bars->p_empty[x]), (x_done + mine - 1) & 1);
                tc_fence_after();
                const int64_t t = ts + tr;
                const T* gate = reinterpret_cast<const T*>(p.gate);
                float f = 0.f;
                if (live) {
                    f = p.out_scale / l;
                    if (EXT && p.gate_per_head && gate != nullptr) f *= 1.f / (1.f + __expf(-ldf(gate + t * p.gate_st + h)));
                }
                const bool stored = live && (solo < 0 || tr == solo);
                float2 odd = make_float2(0.f, 0.f);       // NaN once an entry of O is not finite
                auto look = [&](uint32_t a, uint32_t b) { odd = fma2(make_float2(__uint_as_float(a), __uint_as_float(b)), make_float2(0.f, 0.f), odd); };
                const bool gated = gate != nullptr && !(EXT && p.gate_per_head);
                const T* grow = gated ? gate + t * p.gate_st + (int64_t)h * dv : nullptr;
                const int64_t at = t * p.out_st + (int64_t)h * dv;
                auto gate8 = [&](const Vec8<T>& u, float (&y)[8]) {
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float2 q = gate_pair(make_float2(y[2 * e], y[2 * e + 1]), Traits<T>::to_f2(u.v[e]));
                        y[2 * e] = q.x; y[2 * e + 1] = q.y;
                    }
                };
                auto store8 = [&](int64_t to, float (&y)[8]) {
                    if (p.out_f32) {
                        float* o = reinterpret_cast<float*>(p.out) + to;
                        if (p.out_vec) {
                            *reinterpret_cast<float4*>(o) = make_float4(y[0], y[1], y[2], y[3]);
                            *reinterpret_cast<float4*>(o + 4) = make_float4(y[4], y[5], y[6], y[7]);
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; e++) o[e] = y[e];
                        }
                    } else {
                        T* o = reinterpret_cast<T*>(p.out) + to;
                        if (p.out_vec) {
                            *reinterpret_cast<uint4*>(o) = make_uint4(pack2<T>(y[0], y[1]), pack2<T>(y[2], y[3]), pack2<T>(y[4], y[5]), pack2<T>(y[6], y[7]));
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; e++) stf(o + e, y[e]);
                        }
                    }
                };
                auto put8 = [&](int d, float (&y)[8]) {                            // eight neighbouring entries of this thread's row
                    if (gated) {
                        if (p.gate_vec) {
                            gate8(ld_vec8(grow + d), y);
                        } else {
#pragma unroll
                            for (int e = 0; e < 8; e++) y[e] *= 1.f / (1.f + __expf(-ldf(grow + d + e)));
                        }
                    }
                    store8(at + d, y);
                };
                if (p.vcos == nullptr && p.out_vec && (!gated || p.gate_vec)) {
                    // 64 columns at a time through this tile's query buffer (its products are done), so that a row's gate and output move
                    // as whole lines: eight lanes a row, rows swizzled by 16 bytes
                    float* xs = reinterpret_cast<float*>(q_sm + x * WX_Q_BYTES);
                    auto cell = [&](int rr, int quarter) { return reinterpret_cast<float4*>(xs + rr * 64 + ((quarter ^ (rr & 15)) << 2)); };
                    const int l8 = lane & 7;
                    // this lane's part of row 32 quad + 4 i + lane / 8, where there is something to store: its token and head
                    uint32_t there = 0;
                    int64_t gate_at[8], out_at[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int rr = quad * 32 + 4 * i + (lane >> 3), rt = x * tpt + (rr >> p.hqp_log2), rh = rr & (hqp - 1);
                        const bool is = rt < n && rh < hq && (solo < 0 || rt == solo);
                        const int64_t col = (int64_t)(g * hq + rh) * dv + 8 * l8;
                        there |= is ? 1u << i : 0u;
                        gate_at[i] = is ? (ts + rt) * p.gate_st + col : 0; out_at[i] = is ? (ts + rt) * p.out_st + col : 0;
                    }
                    // (no branches between one row's numbers and the next one's: the rows' exponentials and quotients run side by side)
                    auto rows = [&](auto to_f32, auto with_gate) {
#pragma unroll 1
                        for (int d0 = 0; d0 < dv; d0 += 64) {
                            const bool here = d0 + 8 * l8 < dv;
                            Vec8<T> z[8];             // all gates of the pass are asked for before the first is used
                            if constexpr (with_gate.value) {
#pragma unroll
                                for (int i = 0; i < 8; i++) z[i] = ld_vec8(gate + (here ? gate_at[i] + d0 : 0));
                            }
                            const int cols = min(64, dv - d0);
#pragma unroll 1
                            for (int d = 0; d < cols; d += 16) {
                                uint32_t v[16];
                                tmem_ld<16>(o_addr + d0 + d, v);
                                tmem_ld_wait();
#pragma unroll
                                for (int e = 0; e < 16; e += 2) look(v[e], v[e + 1]);
#pragma unroll
                                for (int e = 0; e < 4; e++)
                                    *cell(row, (d >> 2) + e) = make_float4(__uint_as_float(v[4 * e]) * f, __uint_as_float(v[4 * e + 1]) * f,
                                                                           __uint_as_float(v[4 * e + 2]) * f, __uint_as_float(v[4 * e + 3]) * f);
                            }
                            __syncwarp();             // a warp reads the rows that it wrote
#pragma unroll
                            for (int i0 = 0; i0 < 8; i0 += 4) {
                                float y[4][8];
#pragma unroll
                                for (int k = 0; k < 4; k++) {
                                    const int rr = quad * 32 + 4 * (i0 + k) + (lane >> 3);
                                    const float4 lo4 = *cell(rr, 2 * l8), hi4 = *cell(rr, 2 * l8 + 1);
                                    y[k][0] = lo4.x; y[k][1] = lo4.y; y[k][2] = lo4.z; y[k][3] = lo4.w;
                                    y[k][4] = hi4.x; y[k][5] = hi4.y; y[k][6] = hi4.z; y[k][7] = hi4.w;
                                    if constexpr (with_gate.value) gate8(z[i0 + k], y[k]);
                                }
#pragma unroll
                                for (int k = 0; k < 4; k++) {
                                    if (!here || !(there >> (i0 + k) & 1)) continue;
                                    if constexpr (to_f32.value) {
                                        float* o = reinterpret_cast<float*>(p.out) + out_at[i0 + k] + d0;
                                        *reinterpret_cast<float4*>(o) = make_float4(y[k][0], y[k][1], y[k][2], y[k][3]);
                                        *reinterpret_cast<float4*>(o + 4) = make_float4(y[k][4], y[k][5], y[k][6], y[k][7]);
                                    } else {
                                        *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + out_at[i0 + k] + d0) =
                                            make_uint4(pack2<T>(y[k][0], y[k][1]), pack2<T>(y[k][2], y[k][3]), pack2<T>(y[k][4], y[k][5]), pack2<T>(y[k][6], y[k][7]));
                                    }
                                }
                            }
                            __syncwarp();
                        }
                    };
                    using Yes = std::true_type; using No = std::false_type;
                    if (p.out_f32) { if (gated) rows(Yes(), Yes()); else rows(Yes(), No()); }
                    else if (gated) rows(No(), Yes());
                    else rows(No(), No());
                } else {
                const int hv = dv >> 1;
#pragma unroll 1
                for (int m = 0; m < hv; m += 8) {     // entries m .. m + 7 and m + hv .. (pairs of halves), or 2 m .. 2 m + 15
                    const bool split = p.vcos != nullptr && p.halves;
                    const int da = split ? m : 2 * m, db = split ? m + hv : 2 * m + 8;
                    uint32_t ua[8], ub[8];
                    __syncwarp();
                    tmem_ld<8>(o_addr + da, ua);
                    tmem_ld<8>(o_addr + db, ub);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 8; e += 2) { look(ua[e], ua[e + 1]); look(ub[e], ub[e + 1]); }
                    if (stored) {
                        float a[8], b[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) { a[e] = __uint_as_float(ua[e]) * f; b[e] = __uint_as_float(ub[e]) * f; }
                        if (p.vcos != nullptr) {      // values were stored turned by their position: turned back by the query's
                            const float* vc = p.vcos + t * hv + m;
                            const float* vs = p.vsin + t * hv + m;
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const float cs = vc[e], sn = vs[e];
                                float& u = split ? a[e] : (e < 4 ? a[2 * e] : b[2 * e - 8]);
                                float& w = split ? b[e] : (e < 4 ? a[2 * e + 1] : b[2 * e - 7]);
                                const float u0 = u, w0 = w;
                                u = u0 * cs + w0 * sn; w = w0 * cs - u0 * sn;
                            }
                        }
                        put8(da, a);
                        put8(db, b);
                    }
                }
                __syncwarp();
                }
                // (a row whose sum is NaN is NaN by its own keys)
                if (live && n > 1 && solo < 0 && l == l && odd.x + odd.y != 0.f) tainted[0] = pass;
            }
            tc_fence_before();
            __syncthreads();                          // the next segment overwrites the queries; its first products overwrite O
            tc_fence_after();
            n_done += nsteps; done_a += sg.steps_a; done_b += sg.steps_b;
            if (!again(sg, true)) i0 += n;
        }
    }
    if (warp == 1) tmem_dealloc<512>(tmem);
}

// Heads of fewer than 128 entries in all stay with mma.sync, whose smaller tiles suit them better (16 + 48: 55 against 59 us for four prompts
// of 2048, 21 against 27 for 16 rows at 1500; 64 + 64: 399 against 274 and 74 against 66)
bool window_tc_supported(int dk, int dv, int krot, int hq, float scale, const void* cache, int64_t num_rows) {
    return dk + dv >= 128 && dk % 16 == 0 && dv % 16 == 0 && dk <= 128 && dv <= 128 && krot % 16 == 0 && dk + krot <= 256 && hq <= 64 && scale > 0.f &&
           ((uintptr_t)cache & 15) == 0 && num_rows < (1ll << 31);
}

int launch_window_attn_tc(WindowTc& p, sllm_dtype_t dtype, cudaStream_t stream) {
    const int hq = p.H / p.G;
    p.hqp_log2 = 0;
    while ((1 << p.hqp_log2) < hq) p.hqp_log2++;
    int num_sms = 0;
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, current_device());
    // two full tiles a CTA; fewer tokens (down to half a tile) while all CTAs still find an SM at once: a second round of half-filled ones
    // takes as long as the first (512 rows at 1500, 8 groups: 115 us in 128 CTAs, 211 in 256)
    p.qt = (2 * WX_ROWS) >> p.hqp_log2;
    const int least = (WX_ROWS / 2) >> p.hqp_log2;
    while (p.qt > least && p.qt > 1 && (int64_t)cdiv(p.num_rows, p.qt >> 1) * p.G <= num_sms) p.qt >>= 1;
    const dim3 grid((unsigned)cdiv(p.num_rows, p.qt) * (unsigned)p.G);
    const bool ext = p.slopes != nullptr || p.keep_first > 0 || p.gate_per_head || p.shared_kv || p.sinks != nullptr, cap = p.softcap > 0.f;
    // The long CTAs of all groups first: with one group behind the other the last one's long CTAs begin when most SMs have run out of work (us, one group
    // behind the other / now, three prompts of up to 2048, 16 / 4 heads 74 / 64, 32 / 8 heads at 1000, window 2048 144 / 117, shared keys 181 instead of 229).
    // More than a round of them beside a round of decoded rows keeps the groups apart: those fill the ragged end, and find no SM before the last prompt row's
    // CTA has one (us, apart / together, three prompts of up to 2048 and 38 decoded 83 / 90, 64 decoded 90 / 92, at 300 keys 75 / 76, 32 / 8 heads
    // 178 / 180; less than a round of either, together: ten decoded 83 / 70, one prompt of 1000 58 / 52; shared keys 106 / 100, 216 / 204).  What
    // decides is whether the decoded rows' work fits the ragged end, which their number alone does not say: 64 beside two prompts at 1000, 32 / 8 heads, keep
    // the groups apart and take 147 where together they would take 136
    p.group_blocks = !ext && p.beside >= num_sms && (int64_t)grid.x > num_sms ? cdiv(p.num_rows, p.qt) : 0;
    // boxes: whole cache blocks of 16 rows, 16-byte rows and columns of theirs (a block table names only blocks that there are: the map need not know how
    // many)
    CUtensorMap map = {};
    bool boxes = !ext && p.dk == 128 && p.dv == 128 && p.krot == 0 && p.block_size % 16 == 0 && p.row_elems % 8 == 0 && p.koff % 8 == 0;
    if (boxes) {
        const cuuint64_t dims[2] = {(cuuint64_t)p.row_elems, (cuuint64_t)1 << 31}, strides[1] = {(cuuint64_t)p.row_elems * 2};
        const cuuint32_t box[2] = {64, 16}, es[2] = {1, 1};
        TensorMapEncodeFn enc = get_tensor_map_encoder();
        boxes = enc != nullptr && enc(&map, dtype == SLLM_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p.cache), dims,
                                      strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    }
#define SLLM_WX3(EXT, CAP, FULL, BOXES)                                                                                                          \
    do {                                                                                                                           \
        static unsigned long long configured = 0;                                                                                  \
        auto kern = window_attn_tc_kernel<T, EXT, CAP, FULL, BOXES>;                                                                            \
        if (first_use_on_this_device(configured)) {                                                                                \
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WX_SMEM);                      \
            SLLM_REQUIRE(e == cudaSuccess, "window_attention: cudaFuncSetAttribute: %s", cudaGetErrorString(e));                  \
        }                                                                                                                          \
        launch_early(kern, grid, WX_THREADS, WX_SMEM, stream, map, p);                                                                \
    } while (0)
#define SLLM_WX(EXT, CAP)                                                                                                          \
    do {                                                                                                                           \
        if (!EXT && boxes) SLLM_WX3(EXT, CAP, true, !EXT);                                                                         \
        else if (p.dk == 128 && p.dv == 128 && p.krot == 0) SLLM_WX3(EXT, CAP, true, false);                                       \
        else SLLM_WX3(EXT, CAP, false, false);                                                                                           \
    } while (0)
    SLLM_DISPATCH_DTYPE(dtype, {
        if (ext && cap) SLLM_WX(true, true);
        else if (ext) SLLM_WX(true, false);
        else if (cap) SLLM_WX(false, true);
        else SLLM_WX(false, false);
    });
#undef SLLM_WX
#undef SLLM_WX3
    return check_launch("window_attention (tcgen05)");
}

}  // namespace sllm
