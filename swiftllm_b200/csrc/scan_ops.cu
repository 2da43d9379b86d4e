// Per-channel recurrences over a sequence with per-SEQUENCE state (row `seq` of a state tensor: the sequence's block-table row),
// carried from step to step.  A step brings SEGMENTS: rows seg_starts[b] .. seg_starts[b+1] - 1 of the packed batch are
// consecutive positions of sequence seq_ids[b] (a prompt portion, or one decoded token).  A segment that starts at position 0
// starts from the zero state whatever its row of the state tensor holds (rows are used again without being cleared).
//
//   short_conv         out[t, c] = act(b[c] + sum_k w[c, K-1-k] * x[t-k, c]) (+ x[t, c]); inputs before the segment come from the
//                      sequence's tail (its last K-1 inputs), inputs before position 0 are zero.  Input fp32 or T, output T.
//   conv_tail_update   moves a sequence's tail on by the segment's inputs (runs after every reader of the old tail); a decoded
//                      token's row is the only reader and writer of its sequence's tail, so short_conv moves that tail on itself
//   mingru_scan        z = sigmoid(zl); c = u + 1/2 (u >= 0) | sigmoid(u) (u < 0); S <- (1 - z) S + z c; out = S * silu(g)
//   selective_scan     dt = softplus(dtl + bias); S[c, n] <- exp(dt A[c, n]) S[c, n] + dt x B[n]; y = sum_n S C[n] + D x;
//                      out = y * silu(z)
// Gates, step sizes, decays and the states run in fp32 for every storage type T of the projections.
#include "tc_helpers.cuh"
#include "typed_io.cuh"

namespace sllm {

constexpr int SC_MAX_TAPS = 8;

__device__ __forceinline__ float sigmoid_fn(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_fn(float z) { return z / (1.f + expf(-z)); }
// The same for eight entries at a time: a quotient without a branch, by one step of Newton's iteration for the reciprocal and Markstein's
// correction of the quotient by its remainder, which rounds it as the exact one (4 x 2048 tokens x 4096 channels 470 -> 460 us in all).
// The factors of 1/4 keep the reciprocal of a denominator near 2^128 in range.
__device__ __forceinline__ float2 silu_rows(float2 z) {
    constexpr float MOST = 3.402823466e38f;
    const float2 d = make_float2(1.f + expf(-z.x), 1.f + expf(-z.y)), df = make_float2(-fminf(d.x, MOST), -fminf(d.y, MOST));
    const float2 quarter = make_float2(0.25f, 0.25f), d4 = tc::mul2(d, quarter);        // (d = infinity: reciprocal and quotient 0)
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d4.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d4.y));
    r = tc::mul2(r, quarter);
    r = tc::fma2(r, tc::fma2(df, r, make_float2(1.f, 1.f)), r);
    const float2 q = tc::mul2(z, r);
    const float2 left = tc::fma2(df, q, z);                         // (z = infinity: not a number, and the quotient stands)
    return tc::fma2(make_float2(fminf(left.x, MOST), fminf(left.y, MOST)), r, q);
}
__device__ __forceinline__ float softplus_fn(float z) { return z > 20.f ? z : log1pf(expf(z)); }
// max(z, 0) + log(1 + u), u = e^-|z|, for two entries at a time: log(1 + u) = u + u (u Q(u)), Q of degree 8 from log(1 + u) / u at the Chebyshev
// points of [0, 1] (interpolation error 2^-27), so that the rounding of u Q, which is below 0.31, counts little.  Off 64 bits, in units of
// 2^-24 of the result, z in -12 .. 12: 0.641 in the mean square (log1pf(expf(z)) 0.646; with 1 + u Q as the factor of u 0.675).
__device__ __forceinline__ float2 softplus_rows(float2 z) {
    const float2 u = make_float2(expf(-fabsf(z.x)), expf(-fabsf(z.y)));
    constexpr float c[9] = {-4.999989271e-01f, 3.332971036e-01f, -2.495161593e-01f, 1.966327429e-01f, -1.526966691e-01f, 1.054362357e-01f, -5.637361482e-02f, 1.954252832e-02f, -3.176057013e-03f};
    float2 q = make_float2(c[8], c[8]);
#pragma unroll
    for (int i = 7; i >= 0; i--) q = tc::fma2(q, u, make_float2(c[i], c[i]));
    return tc::add2(tc::fma2(tc::mul2(q, u), u, u), make_float2(fmaxf(z.x, 0.f), fmaxf(z.y, 0.f)));
}
// 2^x for x <= 0 on the special-function unit (relative error about 2^-22; results below the normal range become 0)
__device__ __forceinline__ float exp2_neg(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float cvt_f(float v) { return v; }
__device__ __forceinline__ float cvt_f(__half v) { return __half2float(v); }
__device__ __forceinline__ float cvt_f(__nv_bfloat16 v) { return __bfloat162float(v); }

// grid (ceil(rows / TOKENS), ceil(C / 128)).  tail: TI [rows, K-1, C] (slot i: the input K-1-i positions before the next one).
// A thread walks TOKENS consecutive rows of one channel with the last K-1 inputs in registers; where a row does not continue the
// row above (another sequence, or the tile's first row) the window is filled again: from the rows above as far as they are the
// sequence's previous positions, from the sequence's tail before that, zeros before position 0.
// TOKENS = 1 with move_tail: every row is a one-token segment of its own sequence; its thread then writes the sequence's new tail.
template <typename TI, typename TO, int TOKENS>
__global__ void __launch_bounds__(128) short_conv_kernel(const TI* __restrict__ xin, int64_t xin_stride, const float* __restrict__ w,
                                                         const float* __restrict__ bias, TI* tail,
                                                         const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                                                         TO* __restrict__ out, int64_t row0, int64_t row_end, int C, int K,
                                                         int add_input, int act_silu, int move_tail) {
    const int64_t tile0 = row0 + (int64_t)blockIdx.x * TOKENS;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= C) return;
    float wk[SC_MAX_TAPS], hist[SC_MAX_TAPS];           // wk[k]: weight of the input k positions back; hist[k - 1]: that input
#pragma unroll
    for (int k = 0; k < SC_MAX_TAPS; k++) { wk[k] = k < K ? w[(int64_t)c * K + (K - 1 - k)] : 0.f; hist[k] = 0.f; }
    const float b0 = bias != nullptr ? bias[c] : 0.f;
    const int nrows = (int)min((int64_t)TOKENS, row_end - tile0);
    float xv[TOKENS];
#pragma unroll
    for (int i = 0; i < TOKENS; i++) xv[i] = i < nrows ? ldf(xin + (tile0 + i) * xin_stride + c) : 0.f;
    int prev_seq = -1, prev_pos = -2;
#pragma unroll
    for (int i = 0; i < TOKENS; i++) {
        if (i >= nrows) break;
        const int64_t t = tile0 + i;
        const int seq = tok_seq[t], pos = tok_pos[t];
        if (i == 0 || seq != prev_seq || pos != prev_pos + 1) {
            int above = 0;                              // rows above this one that are the sequence's previous positions
            while (above < K - 1 && t - above - 1 >= 0 && tok_seq[t - above - 1] == seq && tok_pos[t - above - 1] == pos - above - 1) above++;
#pragma unroll
            for (int k = 1; k < SC_MAX_TAPS; k++) {
                float v = 0.f;
                if (k < K && pos - k >= 0)
                    v = k <= above ? ldf(xin + (t - k) * xin_stride + c)
                                   : ldf(tail + ((int64_t)seq * (K - 1) + (K - 1 - (k - above))) * C + c);
                hist[k - 1] = v;
            }
        }
        float acc = b0 + wk[0] * xv[i];
#pragma unroll
        for (int k = 1; k < SC_MAX_TAPS; k++) acc += wk[k] * hist[k - 1];
        if (act_silu) acc = silu_fn(acc);
        if (add_input) acc += xv[i];
        stf(out + t * C + c, acc);
#pragma unroll
        for (int k = SC_MAX_TAPS - 1; k >= 1; k--) hist[k] = hist[k - 1];
        hist[0] = xv[i];
        prev_seq = seq; prev_pos = pos;
        if (TOKENS == 1 && move_tail) {                 // slot i <- the input K - 2 - i positions back (zeros before position 0)
            TI* tl = tail + (int64_t)seq * (K - 1) * C + c;
#pragma unroll
            for (int k = 0; k < SC_MAX_TAPS - 1; k++)
                if (k < K - 1) stf(tl + (int64_t)(K - 2 - k) * C, hist[k]);
        }
    }
}

// The same for prompt rows where rows are whole pieces of four channels: a thread walks SV_TOKENS rows of four neighbouring channels, two at a
// time in packed arithmetic, the next four rows' loads in flight beside the four it works on (wider pieces need 154 registers and leave
// ten warps on an SM: 96 us; eight rows 60, two 58); where the rows of the tile break (another sequence) is found once per warp.  The
// products, their order and the SiLU's value are those above (a quicker quotient turns some roundings, which a state behind the
// convolution keeps).  Bound: bytes, of which enough are in flight only with many warps.  Measured on B200, bf16, 8192 rows x 4096 channels,
// 4 taps: 179 us by the kernel above; a channel's SiLU with a branch, sixteen rows, loads after the work on the rows before them 75;
// now 54.
template <typename TI, typename TO, int K, int SV_TOKENS>
__global__ void __launch_bounds__(128) short_conv_vec_kernel(const TI* __restrict__ xin, int64_t xin_stride, const float* __restrict__ w,
                                                             const float* __restrict__ bias, const TI* __restrict__ tail,
                                                             const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                                                             TO* __restrict__ out, int64_t row_end, int C, int add_input, int act_silu) {
    constexpr int VW = 4, H = K - 1;
    struct alignas(VW * sizeof(TI)) In { TI e[VW]; };
    struct alignas(VW * sizeof(TO)) Out { TO e[VW]; };
    const int64_t tile0 = (int64_t)blockIdx.x * SV_TOKENS;
    const int c = (blockIdx.y * blockDim.x + threadIdx.x) * VW, lane = threadIdx.x & 31;
    const int nrows = (int)min((int64_t)SV_TOKENS, row_end - tile0);
    // bit i of the two: row tile0 - H + i continues the row above it (bits H .. H + SV_TOKENS - 1 are the tile's own rows)
    uint32_t goes_on[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int64_t t = tile0 - H + lane + 32 * q;
        const bool in = t > 0 && t < row_end && t < tile0 + SV_TOKENS;
        goes_on[q] = __ballot_sync(0xffffffffu, in && tok_seq[in ? t : 0] == tok_seq[in ? t - 1 : 0] && tok_pos[in ? t : 0] == tok_pos[in ? t - 1 : 0] + 1);
    }
    const bool live = c < C;
    const int cc = live ? c : 0;
    const TI* col = xin + cc;
    constexpr int AT_ONCE = 4;                          // rows whose loads are in flight together
    In cur[AT_ONCE], next[AT_ONCE];
    auto load = [&](int i0, In (&to)[AT_ONCE]) {
        const TI* at = col + (tile0 + i0) * xin_stride;
#pragma unroll
        for (int u = 0; u < AT_ONCE; u++, at += xin_stride)
            if (i0 + u < nrows) to[u] = *reinterpret_cast<const In*>(at);
    };
    load(0, cur);
    float2 wk[K][VW / 2], b0[VW / 2];                   // two channels at a time: packed arithmetic
#pragma unroll
    for (int e = 0; e < VW; e++) {
        float* b = &b0[e / 2].x + (e & 1);
        *b = bias != nullptr ? bias[cc + e] : 0.f;
        if (K == 4) {
            const float4 f = *reinterpret_cast<const float4*>(w + (int64_t)(cc + e) * 4);
            const float taps[4] = {f.w, f.z, f.y, f.x};
#pragma unroll
            for (int k = 0; k < K; k++) (&wk[k][e / 2].x)[e & 1] = taps[k];
        } else {
#pragma unroll
            for (int k = 0; k < K; k++) (&wk[k][e / 2].x)[e & 1] = w[(int64_t)(cc + e) * K + (K - 1 - k)];
        }
    }
    float2 hist[H][VW / 2];                             // hist[k - 1]: the input k positions back
#pragma unroll
    for (int k = 0; k < H; k++)
#pragma unroll
        for (int e = 0; e < VW / 2; e++) hist[k][e] = make_float2(0.f, 0.f);
    auto refill = [&](int i, uint32_t on) {             // the window of row i, which does not go on from the row before it in registers
        const int64_t t = tile0 + i;                    // (on: goes_on from row i - H on)
        const int seq = tok_seq[t], pos = tok_pos[t];
        int above = 0;                                  // rows above this one that are the sequence's previous positions
        while (above < H && ((on >> (H - above)) & 1)) above++;
#pragma unroll
        for (int k = 1; k <= H; k++) {
            if (pos - k < 0) {
#pragma unroll
                for (int e = 0; e < VW / 2; e++) hist[k - 1][e] = make_float2(0.f, 0.f);
            } else {
                const In v = *reinterpret_cast<const In*>(k <= above ? col + (t - k) * xin_stride : tail + ((int64_t)seq * H + (H - (k - above))) * C + cc);
#pragma unroll
                for (int e = 0; e < VW / 2; e++) hist[k - 1][e] = make_float2(cvt_f(v.e[2 * e]), cvt_f(v.e[2 * e + 1]));
            }
        }
    };
#pragma unroll 1
    for (int i0 = 0; i0 < nrows; i0 += AT_ONCE) {
        load(i0 + AT_ONCE, next);
#pragma unroll
        for (int u = 0; u < AT_ONCE; u++) {
            const int i = i0 + u;
            if (i >= nrows) break;
            if (i == 0 || !((goes_on[0] >> (H + u)) & 1)) refill(i, goes_on[0] >> u);
            Out o;
#pragma unroll
            for (int e = 0; e < VW / 2; e++) {
                const float2 x = make_float2(cvt_f(cur[u].e[2 * e]), cvt_f(cur[u].e[2 * e + 1]));
                float2 acc = tc::fma2(wk[0][e], x, b0[e]);
#pragma unroll
                for (int k = 1; k < K; k++) acc = tc::fma2(wk[k][e], hist[k - 1][e], acc);
                if (act_silu) acc = silu_rows(acc);
                if (add_input) acc = tc::add2(acc, x);
                stf(&o.e[2 * e], acc.x);
                stf(&o.e[2 * e + 1], acc.y);
#pragma unroll
                for (int k = H - 1; k >= 1; k--) hist[k][e] = hist[k - 1][e];
                hist[0][e] = x;
            }
            if (live) *reinterpret_cast<Out*>(out + (tile0 + i) * C + c) = o;
        }
#pragma unroll
        for (int u = 0; u < AT_ONCE; u++) cur[u] = next[u];
        goes_on[0] = __funnelshift_r(goes_on[0], goes_on[1], AT_ONCE);
        goes_on[1] >>= AT_ONCE;
    }
}

// One thread per (segment, channel): tail slot i <- the input at position p0 + n - (K-1) + i, taken from the segment's rows, from
// the old tail, or zero before position 0.
template <typename TI>
__global__ void __launch_bounds__(128) conv_tail_update_kernel(const TI* __restrict__ xin, int64_t xin_stride, TI* __restrict__ tail,
                                                               const int* __restrict__ seg_starts, const int* __restrict__ seq_ids,
                                                               const int* __restrict__ tok_pos, int C, int K) {
    const int b = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int t0 = seg_starts[b], n = seg_starts[b + 1] - t0;
    if (c >= C || n <= 0) return;
    const int seq = seq_ids[b], p0 = tok_pos[t0];
    float old[SC_MAX_TAPS];
    TI* tl = tail + (int64_t)seq * (K - 1) * C + c;
    for (int i = 0; i < K - 1; i++) old[i] = p0 > 0 ? ldf(tl + (int64_t)i * C) : 0.f;
    for (int i = 0; i < K - 1; i++) {
        const int rel = n - (K - 1) + i;                // position relative to the segment's start
        float v = 0.f;
        if (rel >= 0) v = ldf(xin + (int64_t)(t0 + rel) * xin_stride + c);
        else if (p0 + rel >= 0) v = old[rel + K - 1];
        stf(tl + (int64_t)i * C, v);
    }
}

// grid (segments, ceil(C / 128)): one thread per (segment, channel) walks the segment's rows.
// proj: [T, >= 3 C] rows [z logits | candidate pre-activations | output-gate pre-activations] (biases already added).
template <typename T>
__global__ void __launch_bounds__(128) mingru_scan_kernel(const T* __restrict__ proj, int64_t stride, float* __restrict__ state,
                                                          const int* __restrict__ seg_starts, const int* __restrict__ seq_ids,
                                                          const int* __restrict__ tok_pos, T* __restrict__ out, int C) {
    const int b = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    const int t0 = seg_starts[b], n = seg_starts[b + 1] - t0;
    if (c >= C || n <= 0) return;
    const int seq = seq_ids[b];
    float S = tok_pos[t0] > 0 ? state[(int64_t)seq * C + c] : 0.f;
    const T* pr = proj + (int64_t)t0 * stride + c;
    // the loads of the next row are issued before this row's arithmetic
    float zl = ldf(pr), u = ldf(pr + C), g = ldf(pr + 2 * C);
    for (int i = 0; i < n; i++) {
        float zl2 = 0.f, u2 = 0.f, g2 = 0.f;
        if (i + 1 < n) {
            const T* nx = pr + (int64_t)(i + 1) * stride;
            zl2 = ldf(nx); u2 = ldf(nx + C); g2 = ldf(nx + 2 * C);
        }
        const float z = sigmoid_fn(zl);
        const float cand = u >= 0.f ? u + 0.5f : sigmoid_fn(u);
        S = (1.f - z) * S + z * cand;
        stf(out + (int64_t)(t0 + i) * C + c, S * silu_fn(g));
        zl = zl2; u = u2; g = g2;
    }
    state[(int64_t)seq * C + c] = S;
}

// The same recurrence for PROMPT PORTIONS, parallel over time as well: grid (segments, ceil(C / 32)), 8 warps.  Lane: channel;
// warp w: tokens 8 w .. 8 w + 7 of the current tile of 64 tokens.  Every thread turns its tokens' logits into the pairs (a, b) of
// S -> a S + b (all loads of a run are issued before its sigmoids), composes its run into one such map, the eight maps of a tile
// meet in shared memory, every warp takes the state at its run's start from the maps before it and replays its run.
template <typename T>
__global__ void __launch_bounds__(256) mingru_scan_tiled_kernel(const T* __restrict__ proj, int64_t stride, float* __restrict__ state,
                                                                const int* __restrict__ seg_starts, const int* __restrict__ seq_ids,
                                                                const int* __restrict__ tok_pos, T* __restrict__ out, int C) {
    __shared__ float sa[8][32], sb[8][32], s0[32];
    const int b = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = blockIdx.y * 32 + lane;
    const int t0 = seg_starts[b], n = seg_starts[b + 1] - t0;
    if (n <= 0) return;                                 // the whole CTA
    const bool live = c < C;
    const int seq = seq_ids[b];
    if (w == 0) s0[lane] = (live && tok_pos[t0] > 0) ? state[(int64_t)seq * C + c] : 0.f;
    float S = 0.f;
    for (int tile0 = 0; tile0 < n; tile0 += 64) {
        const int j0 = tile0 + w * 8;
        float a[8], bb[8], g[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {                   // raw logits first: 24 loads in flight
            const bool ok = live && j0 + j < n;
            const T* pr = proj + (int64_t)(t0 + j0 + j) * stride + c;
            a[j] = ok ? ldf(pr) : 0.f;
            bb[j] = ok ? ldf(pr + C) : 0.f;
            g[j] = ok ? ldf(pr + 2 * C) : 0.f;
        }
        float A = 1.f, B = 0.f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (live && j0 + j < n) {
                const float z = sigmoid_fn(a[j]), u = bb[j];
                a[j] = 1.f - z;
                bb[j] = z * (u >= 0.f ? u + 0.5f : sigmoid_fn(u));
                g[j] = silu_fn(g[j]);
            } else {
                a[j] = 1.f; bb[j] = 0.f;                // past the segment's end: the identity map
            }
            B = a[j] * B + bb[j];
            A *= a[j];
        }
        sa[w][lane] = A; sb[w][lane] = B;
        __syncthreads();
        S = s0[lane];
        for (int k = 0; k < w; k++) S = sa[k][lane] * S + sb[k][lane];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            S = a[j] * S + bb[j];
            if (live && j0 + j < n) stf(out + (int64_t)(t0 + j0 + j) * C + c, S * g[j]);
        }
        __syncthreads();                                // s0 and the maps have been read
        if (w == 7) s0[lane] = S;                       // the tile's last run ends at the tile's end state
    }
    if (w == 7 && live) state[(int64_t)seq * C + c] = S;
}

// Block: 128 threads = (128 / NS) channels x NS lanes per channel; lane s of a channel holds the RE = ceil(N / NS) <= SS_R
// consecutive states n = s RE + r of its channel in registers.  grid (segments, ceil(C / (128 / NS))).  x, z: T [T, C] (row strides); dtl: TD [T, C] step logits (without
// bias); bc: T [T, ...] rows with B at column b_off and C at column c_off (N each); A fp32 [C, N] (negative); state fp32
// [rows, C, N].
constexpr int SS_R = 8;

template <typename T, typename TD>
__global__ void __launch_bounds__(128) selective_scan_kernel(
    const T* __restrict__ x, int64_t x_stride, const TD* __restrict__ dtl, int64_t dt_stride, const float* __restrict__ dt_bias,
    const float* __restrict__ A, const T* __restrict__ bc, int64_t bc_stride, int b_off, int c_off, const float* __restrict__ D,
    const T* __restrict__ z, int64_t z_stride, float* __restrict__ state, const int* __restrict__ seg_starts,
    const int* __restrict__ seq_ids, const int* __restrict__ tok_pos, T* __restrict__ out, int C, int N, int ns_log2) {
    const int NS = 1 << ns_log2, RE = (N + NS - 1) >> ns_log2;
    const int b = blockIdx.x;
    const int s = threadIdx.x & (NS - 1);
    const int c = blockIdx.y * (blockDim.x >> ns_log2) + (threadIdx.x >> ns_log2);
    const int t0 = seg_starts[b], n = seg_starts[b + 1] - t0;
    if (n <= 0) return;
    const bool live = c < C;                            // dead threads still take part in the shuffles
    const int cc = live ? c : 0;
    const int seq = seq_ids[b];
    const bool fresh = tok_pos[t0] == 0;
    float S[SS_R], a[SS_R];
    float* sp = state + ((int64_t)seq * C + cc) * N;
#pragma unroll
    for (int r = 0; r < SS_R; r++) {
        const int k = s * RE + r;
        const bool ok = r < RE && k < N;
        a[r] = ok ? A[(int64_t)cc * N + k] * 1.4426950408889634f : 0.f;       // exp(dt A) = 2^(dt A log2 e)
        S[r] = (ok && !fresh) ? sp[k] : 0.f;
    }
    const float bias = dt_bias[cc], dd = D[cc];
    for (int i = 0; i < n; i++) {
        const int64_t t = t0 + i;
        const float dt = softplus_fn(ldf(dtl + t * dt_stride + cc) + bias);
        const float xv = ldf(x + t * x_stride + cc);
        const float dx = dt * xv;
        const T* br = bc + t * bc_stride;
        float y = 0.f;
#pragma unroll
        for (int r = 0; r < SS_R; r++) {
            const int k = s * RE + r;
            if (r < RE && k < N) {
                S[r] = exp2_neg(dt * a[r]) * S[r] + dx * ldf(br + b_off + k);
                y += S[r] * ldf(br + c_off + k);
            }
        }
        for (int o = NS >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        if (s == 0 && live) stf(out + t * C + c, (y + dd * xv) * silu_fn(ldf(z + t * z_stride + c)));
    }
    if (live) {
#pragma unroll
        for (int r = 0; r < SS_R; r++) {
            const int k = s * RE + r;
            if (r < RE && k < N) sp[k] = S[r];
        }
    }
}

// The same scan for PROMPT PORTIONS with staged tiles of `tt` tokens (tt * (128 / NS) <= 128 SS_ITEMS: 8 tokens for NS = 1, 16 for
// NS = 2, 32 from NS = 4 on, fewer when the B / C rows of very wide states would not fit): all threads first bring the tile's x, step sizes (softplus
// applied), SiLU gates and B / C rows into shared memory with coalesced loads (one exposed load latency per tile instead of one
// per token), the sequential part then reads shared memory only, and the tile's outputs leave coalesced.  The raw values of the
// NEXT tile are loaded into registers before the sequential part of the current one and are only touched after it, so their
// latency hides behind the arithmetic (B / C rows: the first SS_BCR x 128 entries of a tile; wider states load the rest when
// they stage).  Same thread layout, same arithmetic per step.  Dynamic shared memory: (4 tt (128 / NS) + 2 tt N) floats.
constexpr int SS_ITEMS = 8;
constexpr int SS_BCR = 4;

// VEC (16-bit rows in 16-byte pieces, states in whole eights): a thread brings eight neighbouring channels of ONE token and eight entries of
// B or C per tile, with one address each, and stores eight outputs; staging with an address per entry took 85 of 125 instructions per
// token.  16 states with fp32 step logits have a kernel of their own below.
// N16: 16 states on two lanes, known to the compiler (many short portions, and states that are not aligned; with the shape unknown 1.4
// times as long).
template <typename T, typename TD, bool VEC, bool N16 = false>
__global__ void __launch_bounds__(128) selective_scan_tiled_kernel(
    const T* __restrict__ x, int64_t x_stride, const TD* __restrict__ dtl, int64_t dt_stride, const float* __restrict__ dt_bias,
    const float* __restrict__ A, const T* __restrict__ bc, int64_t bc_stride, int b_off, int c_off, const float* __restrict__ D,
    const T* __restrict__ z, int64_t z_stride, float* __restrict__ state, const int* __restrict__ seg_starts,
    const int* __restrict__ seq_ids, const int* __restrict__ tok_pos, T* __restrict__ out, int C, int N_, int ns_log2_, int tt_) {
    extern __shared__ __align__(16) float ssm[];
    const int N = N16 ? 16 : N_, ns_log2 = N16 ? 1 : ns_log2_, tt = N16 ? 2 * SS_ITEMS : tt_;
    const int NS = 1 << ns_log2, ch_log2 = 7 - ns_log2, CH = 1 << ch_log2, RE = (N + NS - 1) >> ns_log2;
    // whole groups of four states per lane, on 16-byte boundaries of the staged rows: B and C are read four at a time
    const bool vec = (N & 3) == 0 && (RE & 3) == 0;
    float* xs = ssm;                                    // [tt][CH]
    float* ds = xs + tt * CH;
    float* zs = ds + tt * CH;
    float* ys = zs + tt * CH;
    float* bs = ys + tt * CH;                           // [tt][N]
    float* cs = bs + tt * N;
    const int b = blockIdx.x, tid = threadIdx.x;
    const int s = tid & (NS - 1), cl = tid >> ns_log2;
    const int cbase = blockIdx.y * CH, c = cbase + cl;
    const int t0 = seg_starts[b], n = seg_starts[b + 1] - t0;
    if (n <= 0) return;
    const bool live = c < C;
    const int cc = live ? c : 0;
    const int seq = seq_ids[b];
    const bool fresh = tok_pos[t0] == 0;
    float S[SS_R], a[SS_R];
    float* sp = state + ((int64_t)seq * C + cc) * N;
#pragma unroll
    for (int r = 0; r < SS_R; r++) {
        const int k = s * RE + r;
        const bool ok = r < RE && k < N;
        a[r] = ok ? A[(int64_t)cc * N + k] * 1.4426950408889634f : 0.f;       // exp(dt A) = 2^(dt A log2 e)
        S[r] = (ok && !fresh) ? sp[k] : 0.f;
    }
    const float dd = D[cc];
    // item i of a thread: entry tid + 128 i of the tile.  Kept as loaded: a conversion right behind a load would make the warp wait
    // for it before the sequential part instead of after
    alignas(16) T rx[SS_ITEMS], rz[SS_ITEMS], rbc[8];
    T rb[SS_BCR], rc[SS_BCR];
    alignas(16) TD rd[SS_ITEMS];
    struct alignas(16) Piece { T e[8]; };
    struct alignas(16) PieceD { TD e[8]; };
    // VEC: this thread's token and first channel of a tile, its entries of B (bc_idx < 0) or C
    const int vj = tid >> (ch_log2 >= 3 ? ch_log2 - 3 : 0), vc = (tid & ((CH >> 3) - 1)) * 8, n8 = N >> 3;
    const bool v_live = VEC && vj < tt && cbase + vc < C;
    const int bcn = tt * n8, bi = VEC && tid >= bcn ? tid - bcn : tid;
    const int bj = VEC ? bi / n8 : 0, bk = VEC ? (bi - bj * n8) * 8 : 0;
    const bool second = VEC && tid >= bcn, bc_live = VEC && tid < 2 * bcn;
    float vbias[8];
    if constexpr (VEC) {
#pragma unroll
        for (int e = 0; e < 8; e++) vbias[e] = v_live ? dt_bias[cbase + vc + e] : 0.f;
    }
    auto fetch = [&](int tile0) {
        const int nt = min(tt, n - tile0);                              // <= 0 past the end: nothing is loaded
        const int64_t tb = t0 + tile0;
        if constexpr (VEC) {
            if (v_live && vj < nt) {
                const int64_t t = tb + vj;
                *reinterpret_cast<Piece*>(rx) = *reinterpret_cast<const Piece*>(x + t * x_stride + cbase + vc);
                *reinterpret_cast<PieceD*>(rd) = *reinterpret_cast<const PieceD*>(dtl + t * dt_stride + cbase + vc);
                *reinterpret_cast<Piece*>(rz) = *reinterpret_cast<const Piece*>(z + t * z_stride + cbase + vc);
            }
            if (bc_live && bj < nt) *reinterpret_cast<Piece*>(rbc) = *reinterpret_cast<const Piece*>(bc + (tb + bj) * bc_stride + (second ? c_off : b_off) + bk);
            return;
        }
#pragma unroll
        for (int i = 0; i < SS_ITEMS; i++) {
            const int idx = tid + 128 * i, j = idx >> ch_log2, cg = cbase + (idx & (CH - 1));
            if (idx < (nt << ch_log2) && cg < C) {
                rx[i] = x[(tb + j) * x_stride + cg];
                rd[i] = dtl[(tb + j) * dt_stride + cg];
                rz[i] = z[(tb + j) * z_stride + cg];
            }
        }
#pragma unroll
        for (int i = 0; i < SS_BCR; i++) {
            const int idx = tid + 128 * i;
            if (idx < nt * N) {
                const int j = idx / N, k = idx - j * N;
                const T* br = bc + (tb + j) * bc_stride;
                rb[i] = br[b_off + k];
                rc[i] = br[c_off + k];
            }
        }
    };
    fetch(0);
    for (int tile0 = 0; tile0 < n; tile0 += tt) {
        const int nt = min(tt, n - tile0);
        const int64_t tb = t0 + tile0;
        if constexpr (VEC) {
            auto put = [&](float* to, const float (&v)[8]) {
                reinterpret_cast<float4*>(to)[0] = make_float4(v[0], v[1], v[2], v[3]);
                reinterpret_cast<float4*>(to)[1] = make_float4(v[4], v[5], v[6], v[7]);
            };
            if (v_live && vj < nt) {
                float f[8];
                const int at = (vj << ch_log2) + vc;
#pragma unroll
                for (int e = 0; e < 8; e++) f[e] = cvt_f(rx[e]);
                put(xs + at, f);
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float2 y = softplus_rows(make_float2(cvt_f(rd[e]) + vbias[e], cvt_f(rd[e + 1]) + vbias[e + 1]));
                    f[e] = y.x; f[e + 1] = y.y;
                }
                put(ds + at, f);
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float2 y = silu_rows(make_float2(cvt_f(rz[e]), cvt_f(rz[e + 1])));
                    f[e] = y.x; f[e + 1] = y.y;
                }
                put(zs + at, f);
            }
            auto stage_bc = [&](const T* from, int j, int k, bool of_c) {
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; e++) f[e] = cvt_f(from[e]);
                put((of_c ? cs : bs) + j * N + k, f);
            };
            if (bc_live && bj < nt) stage_bc(rbc, bj, bk, second);
            for (int i = tid + 128; i < 2 * bcn; i += 128) {             // very wide states
                const bool of_c = i >= bcn;
                const int ii = of_c ? i - bcn : i, j = ii / n8, k = (ii - j * n8) * 8;
                if (j < nt) {
                    alignas(16) T v[8];
                    *reinterpret_cast<Piece*>(v) = *reinterpret_cast<const Piece*>(bc + (tb + j) * bc_stride + (of_c ? c_off : b_off) + k);
                    stage_bc(v, j, k, of_c);
                }
            }
        } else {
#pragma unroll
        for (int i = 0; i < SS_ITEMS; i++) {
            const int idx = tid + 128 * i, cg = cbase + (idx & (CH - 1));
            if (idx < (nt << ch_log2) && cg < C) {
                xs[idx] = cvt_f(rx[i]);
                ds[idx] = softplus_fn(cvt_f(rd[i]) + dt_bias[cg]);
                zs[idx] = silu_fn(cvt_f(rz[i]));
            }
        }
#pragma unroll
        for (int i = 0; i < SS_BCR; i++) {
            const int idx = tid + 128 * i;
            if (idx < nt * N) { bs[idx] = cvt_f(rb[i]); cs[idx] = cvt_f(rc[i]); }
        }
        for (int idx = tid + 128 * SS_BCR; idx < nt * N; idx += 128) {
            const int j = idx / N, k = idx - j * N;
            const T* br = bc + (tb + j) * bc_stride;
            bs[idx] = ldf(br + b_off + k);
            cs[idx] = ldf(br + c_off + k);
        }
        }
        __syncthreads();
        fetch(tile0 + tt);                              // in flight during the sequential part below
        const float* bp = bs + s * RE;
        const float* cp = cs + s * RE;
        const bool lane_live = s * RE < N;
        if (N16 || (vec && ns_log2 >= 2 && (tt & 3) == 0)) {
            // four tokens at a time, packed arithmetic; the four sums over the lanes of a channel are taken together, each lane quarter
            // keeping the token (2 (s & 1) + (s >> 1 & 1)) that it writes
            auto four = [&](int j, bool whole) {        // tokens j .. j + 3 (those below nt)
                float y[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    y[u] = 0.f;
                    if (whole || j + u < nt) {
                        const float dt = ds[((j + u) << ch_log2) + cl], dx = dt * xs[((j + u) << ch_log2) + cl];
                        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                        for (int q = 0; q < SS_R / 4; q++) {
                            if (N16 || (4 * q < RE && lane_live)) {
                                const float4 b4 = reinterpret_cast<const float4*>(bp + (j + u) * N)[q], c4 = reinterpret_cast<const float4*>(cp + (j + u) * N)[q];
                                float2 s0 = make_float2(S[4 * q], S[4 * q + 1]), s1 = make_float2(S[4 * q + 2], S[4 * q + 3]);
                                const float2 e0 = make_float2(exp2_neg(dt * a[4 * q]), exp2_neg(dt * a[4 * q + 1]));
                                const float2 e1 = make_float2(exp2_neg(dt * a[4 * q + 2]), exp2_neg(dt * a[4 * q + 3]));
                                s0 = tc::fma2(e0, s0, make_float2(dx * b4.x, dx * b4.y));
                                s1 = tc::fma2(e1, s1, make_float2(dx * b4.z, dx * b4.w));
                                acc = tc::fma2(s0, make_float2(c4.x, c4.y), acc);
                                acc = tc::fma2(s1, make_float2(c4.z, c4.w), acc);
                                S[4 * q] = s0.x; S[4 * q + 1] = s0.y; S[4 * q + 2] = s1.x; S[4 * q + 3] = s1.y;
                            }
                        }
                        y[u] = acc.x + acc.y;
                    }
                }
                const bool odd = s & 1, high = s & 2;
                const float k0 = odd ? y[2] : y[0], k1 = odd ? y[3] : y[1];                          // kept pair
                const float p0 = k0 + __shfl_xor_sync(0xffffffffu, odd ? y[0] : y[2], 1), p1 = k1 + __shfl_xor_sync(0xffffffffu, odd ? y[1] : y[3], 1);
                if constexpr (N16) {
                    const int mine = j + 2 * (s & 1), at = (mine << ch_log2) + cl;
                    if (whole || mine < nt) ys[at] = (p0 + dd * xs[at]) * zs[at];
                    if (whole || mine + 1 < nt) ys[at + CH] = (p1 + dd * xs[at + CH]) * zs[at + CH];
                } else {
                    float v = (high ? p1 : p0) + __shfl_xor_sync(0xffffffffu, high ? p0 : p1, 2);
                    for (int o = NS >> 1; o > 2; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    const int mine = j + 2 * (s & 1) + ((s >> 1) & 1);
                    if (s < 4 && (whole || mine < nt)) {
                        const int at = (mine << ch_log2) + cl;
                        ys[at] = (v + dd * xs[at]) * zs[at];
                    }
                }
            };
            if (nt == tt) {
#pragma unroll 2
                for (int j = 0; j < tt; j += 4) four(j, true);
            } else {
                for (int j = 0; j < nt; j += 4) four(j, false);
            }
        } else
        for (int j = 0; j < nt; j++, bp += N, cp += N) {
            const float dt = ds[(j << ch_log2) + cl], xv = xs[(j << ch_log2) + cl];
            const float dx = dt * xv;
            float y = 0.f;
            if (vec) {
#pragma unroll
                for (int q = 0; q < SS_R / 4; q++) {
                    if (4 * q < RE && lane_live) {
                        const float4 b4 = reinterpret_cast<const float4*>(bp)[q], c4 = reinterpret_cast<const float4*>(cp)[q];
                        S[4 * q + 0] = exp2_neg(dt * a[4 * q + 0]) * S[4 * q + 0] + dx * b4.x;
                        S[4 * q + 1] = exp2_neg(dt * a[4 * q + 1]) * S[4 * q + 1] + dx * b4.y;
                        S[4 * q + 2] = exp2_neg(dt * a[4 * q + 2]) * S[4 * q + 2] + dx * b4.z;
                        S[4 * q + 3] = exp2_neg(dt * a[4 * q + 3]) * S[4 * q + 3] + dx * b4.w;
                        y += S[4 * q + 0] * c4.x + S[4 * q + 1] * c4.y + S[4 * q + 2] * c4.z + S[4 * q + 3] * c4.w;
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < SS_R; r++) {
                    if (r < RE && s * RE + r < N) {
                        S[r] = exp2_neg(dt * a[r]) * S[r] + dx * bp[r];
                        y += S[r] * cp[r];
                    }
                }
            }
            for (int o = NS >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
            if (s == 0) ys[(j << ch_log2) + cl] = (y + dd * xv) * zs[(j << ch_log2) + cl];
        }
        __syncthreads();
        if constexpr (VEC) {
            if (v_live && vj < nt) {
                const float4 lo = *reinterpret_cast<const float4*>(ys + (vj << ch_log2) + vc), hi = *reinterpret_cast<const float4*>(ys + (vj << ch_log2) + vc + 4);
                Piece o;
                stf(o.e, lo.x); stf(o.e + 1, lo.y); stf(o.e + 2, lo.z); stf(o.e + 3, lo.w);
                stf(o.e + 4, hi.x); stf(o.e + 5, hi.y); stf(o.e + 6, hi.z); stf(o.e + 7, hi.w);
                *reinterpret_cast<Piece*>(out + (tb + vj) * C + cbase + vc) = o;
            }
        } else
        for (int idx = tid; idx < (nt << ch_log2); idx += 128) {
            const int j = idx >> ch_log2, cg = cbase + (idx & (CH - 1));
            if (cg < C) stf(out + (tb + j) * C + cg, ys[idx]);
        }
        // the next tile's staging writes xs / ds / zs / bs / cs, which nobody reads any more; ys is written again only after
        // the next barrier
    }
    if (live) {
#pragma unroll
        for (int r = 0; r < SS_R; r++) {
            const int k = s * RE + r;
            if (r < RE && k < N) sp[k] = S[r];
        }
    }
}

// Prompt portions of 16 states, 16-bit rows in 16-byte pieces, fp32 step logits: four lanes of four states per channel, CPL neighbouring
// channels per lane.  grid (segments, ceil(C / (32 CPL))), four WALKERS that go through the tokens, and 4 CPL STAGERS, a tile of 32 tokens ahead
// and one behind: a stager's thread brings eight neighbouring channels of a token, turns the step logits into
// steps and leaves dt and dt x; once the walkers have left the sums over the states it adds D x, applies the gate and stores.  The rows
// after next are asked for before that.
// Bound: issue and the special-function unit (16 powers and 5 more results per token and channel: 150 us at the size below), once
// nothing waits: with the same threads staging and walking in turn 325 us, at 0.39 instructions per cycle.  B and C are 128 bytes per
// token and channel from shared memory, which gives 128 a cycle: two channels per lane share them where there are warps enough; beyond
// that (more powers by polynomial instead of the special-function unit: 275 us) nothing gave.  Measured on B200,
// bf16, 4 x 2048 tokens, 4096 channels: 380 -> 247 us; one segment of 1024 tokens 122 -> 59.
constexpr int SP_TILE = 32;
template <int CPL> struct SpSmem {
    static constexpr int CH = 32 * CPL, YP = CH + 8 * CPL;              // channels; floats between rows of y (no bank conflicts)
    struct Tile {
        float dt[SP_TILE * CH], dx[SP_TILE * CH], y[SP_TILE * YP], b[SP_TILE * 16], c[SP_TILE * 16];
        uint4 x[128 * CPL], z[128 * CPL];                               // pieces as loaded, for the thread that brought them
    } tile[2];
};
template <typename T, int CPL>
__global__ void __launch_bounds__(128 + 128 * CPL, CPL == 1 ? 3 : 2) selective_scan16_kernel(
    const T* __restrict__ x, int64_t x_stride, const float* __restrict__ dtl, int64_t dt_stride, const float* __restrict__ dt_bias,
    const float* __restrict__ A, const T* __restrict__ bc, int64_t bc_stride, int b_off, int c_off, const float* __restrict__ D,
    const T* __restrict__ z, int64_t z_stride, float* __restrict__ state, const int* __restrict__ seg_starts,
    const int* __restrict__ seq_ids, const int* __restrict__ tok_pos, T* __restrict__ out, int C) {
    using Smem = SpSmem<CPL>;
    constexpr int CH = Smem::CH, YP = Smem::YP, PIECES = CH / 8, ALL = 128 + 128 * CPL;    // pieces of a token: one thread each for a tile's
    constexpr int FULL = 1, DONE = 3;                                   // named barriers, one per tile in shared memory
    extern __shared__ __align__(16) unsigned char sp_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(sp_raw);
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, s = lane & 3;
    const int t0 = seg_starts[b], n = seg_starts[b + 1] - t0;
    if (n <= 0) return;
    const int cbase = blockIdx.y * CH;
    if (threadIdx.x >= 128) {
        // ================ stagers: piece vp of token vj; the first four warps also eight entries of B or C of one token
        const int st = tid - 128, vp = (st % PIECES) * 8, vj = st / PIECES, bj = st < 128 ? (st & 63) >> 1 : SP_TILE, bk = (st & 1) * 8;
        const bool v_live = cbase + vp < C, second = st >= 64;
        struct alignas(16) Piece { T e[8]; };
        Piece rx, rz, rb;
        float4 rd[2];
        float bias[8], skip[8];
#pragma unroll
        for (int e = 0; e < 8; e++) { bias[e] = v_live ? dt_bias[cbase + vp + e] : 0.f; skip[e] = v_live ? D[cbase + vp + e] : 0.f; }
        auto fetch = [&](int tile0) {
            const int nt = min(SP_TILE, n - tile0);                     // <= 0 past the end: nothing is loaded
            const int64_t t = t0 + tile0 + vj;
            if (v_live && vj < nt) {
                rx = *reinterpret_cast<const Piece*>(x + t * x_stride + cbase + vp);
                rz = *reinterpret_cast<const Piece*>(z + t * z_stride + cbase + vp);
                const float4* d = reinterpret_cast<const float4*>(dtl + t * dt_stride + cbase + vp);
                rd[0] = d[0]; rd[1] = d[1];
            }
            if (bj < nt) rb = *reinterpret_cast<const Piece*>(bc + (t0 + tile0 + bj) * bc_stride + (second ? c_off : b_off) + bk);
        };
        auto stage = [&](int tile0) {                                   // what was fetched last
            const int nt = min(SP_TILE, n - tile0), buf = tile0 / SP_TILE & 1;
            typename Smem::Tile& to = sm.tile[buf];
            if (v_live && vj < nt) {
                to.x[st] = *reinterpret_cast<const uint4*>(&rx);
                to.z[st] = *reinterpret_cast<const uint4*>(&rz);
                const float* d = reinterpret_cast<const float*>(rd);
                float f[8], g[8];
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float2 dt = softplus_rows(tc::add2(make_float2(d[e], d[e + 1]), make_float2(bias[e], bias[e + 1])));
                    const float2 v = tc::mul2(dt, make_float2(cvt_f(rx.e[e]), cvt_f(rx.e[e + 1])));
                    f[e] = dt.x; f[e + 1] = dt.y; g[e] = v.x; g[e + 1] = v.y;
                }
#pragma unroll
                for (int e = 0; e < 8; e += 4) {
                    *reinterpret_cast<float4*>(&to.dt[vj * CH + vp + e]) = make_float4(f[e], f[e + 1], f[e + 2], f[e + 3]);
                    *reinterpret_cast<float4*>(&to.dx[vj * CH + vp + e]) = make_float4(g[e], g[e + 1], g[e + 2], g[e + 3]);
                }
            }
            if (bj < nt) {
                float* at = (second ? to.c : to.b) + bj * 16 + bk;
#pragma unroll
                for (int e = 0; e < 8; e += 4)
                    *reinterpret_cast<float4*>(at + e) = make_float4(cvt_f(rb.e[e]), cvt_f(rb.e[e + 1]), cvt_f(rb.e[e + 2]), cvt_f(rb.e[e + 3]));
            }
            tc::named_bar_arrive(FULL + buf, ALL);
        };
        fetch(0);
        stage(0);
        fetch(SP_TILE);
        for (int tile0 = 0; tile0 < n; tile0 += SP_TILE) {
            if (tile0 + SP_TILE < n) {
                stage(tile0 + SP_TILE);                                 // the walkers are done with the tile before this one
                fetch(tile0 + 2 * SP_TILE);
            }
            const int nt = min(SP_TILE, n - tile0), buf = tile0 / SP_TILE & 1;
            const typename Smem::Tile& from = sm.tile[buf];
            tc::named_bar_sync(DONE + buf, ALL);
            if (v_live && vj < nt) {
                Piece px, pz, o;
                *reinterpret_cast<uint4*>(&px) = from.x[st];
                *reinterpret_cast<uint4*>(&pz) = from.z[st];
                const float* y = &from.y[vj * YP + vp];
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float2 g = silu_rows(make_float2(cvt_f(pz.e[e]), cvt_f(pz.e[e + 1])));
                    const float2 w = tc::mul2(tc::fma2(make_float2(skip[e], skip[e + 1]), make_float2(cvt_f(px.e[e]), cvt_f(px.e[e + 1])), *reinterpret_cast<const float2*>(y + e)), g);
                    stf(o.e + e, w.x);
                    stf(o.e + e + 1, w.y);
                }
                *reinterpret_cast<Piece*>(out + (t0 + tile0 + vj) * C + cbase + vp) = o;
            }
        }
        return;
    }
    // ================ walkers
    const int cl = (tid >> 5) * 8 * CPL + (lane >> 2) * CPL;            // this lane's first channel, in the CTA
    const bool fresh = tok_pos[t0] == 0;
    const int64_t row0 = (int64_t)seq_ids[b] * C;
    float2 S[CPL][2], a[CPL][2];
#pragma unroll
    for (int c = 0; c < CPL; c++) {
        const int cc = min(cbase + cl + c, C - 1);                      // channels past the end take part in the shuffles
        const float4 f = *reinterpret_cast<const float4*>(A + (int64_t)cc * 16 + 4 * s);
        constexpr float L = 1.4426950408889634f;                        // exp(dt A) = 2^(dt A log2 e)
        a[c][0] = make_float2(f.x * L, f.y * L); a[c][1] = make_float2(f.z * L, f.w * L);
        const float4 h = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(state + (row0 + cc) * 16 + 4 * s);
        S[c][0] = make_float2(h.x, h.y); S[c][1] = make_float2(h.z, h.w);
    }
    for (int tile0 = 0; tile0 < n; tile0 += SP_TILE) {
        const int nt = min(SP_TILE, n - tile0), buf = tile0 / SP_TILE & 1;
        typename Smem::Tile& tile = sm.tile[buf];
        // four tokens at a time; their sums over a channel's lanes are taken together, lane s keeps token 2 (s & 1) + (s >> 1)
        auto four = [&](int j, bool all) {                              // tokens j .. j + 3 (those below nt)
            float y[4][CPL];
#pragma unroll
            for (int u = 0; u < 4; u++) {
#pragma unroll
                for (int c = 0; c < CPL; c++) y[u][c] = 0.f;
                if (!all && j + u >= nt) continue;
                const float4 b4 = *reinterpret_cast<const float4*>(&tile.b[(j + u) * 16 + 4 * s]), c4 = *reinterpret_cast<const float4*>(&tile.c[(j + u) * 16 + 4 * s]);
                float dt[CPL], dx[CPL];
                if constexpr (CPL == 2) {
                    const float2 d2 = *reinterpret_cast<const float2*>(&tile.dt[(j + u) * CH + cl]), x2 = *reinterpret_cast<const float2*>(&tile.dx[(j + u) * CH + cl]);
                    dt[0] = d2.x; dt[CPL - 1] = d2.y; dx[0] = x2.x; dx[CPL - 1] = x2.y;
                } else {
                    dt[0] = tile.dt[(j + u) * CH + cl]; dx[0] = tile.dx[(j + u) * CH + cl];
                }
#pragma unroll
                for (int c = 0; c < CPL; c++) {
                    const float2 d2 = make_float2(dt[c], dt[c]), x2 = make_float2(dx[c], dx[c]);
                    const float2 p0 = tc::mul2(d2, a[c][0]), p1 = tc::mul2(d2, a[c][1]);
                    S[c][0] = tc::fma2(make_float2(exp2_neg(p0.x), exp2_neg(p0.y)), S[c][0], tc::mul2(x2, make_float2(b4.x, b4.y)));
                    S[c][1] = tc::fma2(make_float2(exp2_neg(p1.x), exp2_neg(p1.y)), S[c][1], tc::mul2(x2, make_float2(b4.z, b4.w)));
                    const float2 acc = tc::fma2(S[c][1], make_float2(c4.z, c4.w), tc::mul2(S[c][0], make_float2(c4.x, c4.y)));
                    y[u][c] = acc.x + acc.y;
                }
            }
            const bool odd = s & 1, high = s & 2;
            float v[CPL];
#pragma unroll
            for (int c = 0; c < CPL; c++) {
                const float p0 = (odd ? y[2][c] : y[0][c]) + __shfl_xor_sync(0xffffffffu, odd ? y[0][c] : y[2][c], 1);
                const float p1 = (odd ? y[3][c] : y[1][c]) + __shfl_xor_sync(0xffffffffu, odd ? y[1][c] : y[3][c], 1);
                v[c] = (high ? p1 : p0) + __shfl_xor_sync(0xffffffffu, high ? p0 : p1, 2);
            }
            float* to = &tile.y[(j + 2 * (s & 1) + (s >> 1)) * YP + cl];                    // rows up to SP_TILE - 1 exist whatever nt
            if constexpr (CPL == 2) *reinterpret_cast<float2*>(to) = make_float2(v[0], v[CPL - 1]);
            else *to = v[0];
        };
        tc::named_bar_sync(FULL + buf, ALL);
        if (nt == SP_TILE) {
#pragma unroll 2
            for (int j = 0; j < SP_TILE; j += 4) four(j, true);
        } else {
            for (int j = 0; j < nt; j += 4) four(j, false);
        }
        tc::named_bar_arrive(DONE + buf, ALL);
    }
#pragma unroll
    for (int c = 0; c < CPL; c++)
        if (cbase + cl + c < C)
            *reinterpret_cast<float4*>(state + (row0 + cbase + cl + c) * 16 + 4 * s) = make_float4(S[c][0].x, S[c][0].y, S[c][1].x, S[c][1].y);
}

}  // namespace sllm

using namespace sllm;

extern "C" {

int sllm_short_conv(const void* xin, int64_t xin_stride, sllm_dtype_t in_dtype, const void* w, const void* bias, const void* tail,
                    const void* tok_seq, const void* tok_pos, void* out, sllm_dtype_t out_dtype, int64_t num_tokens,
                    int64_t num_prefill_tokens, int channels, int taps, int add_input, int act_silu, int move_decode_tails,
                    sllm_stream_t stream) {
    SLLM_REQUIRE(num_tokens >= 0 && channels > 0 && taps >= 1 && taps <= SC_MAX_TAPS, "short_conv: 1 <= taps <= %d (got %d)",
                 SC_MAX_TAPS, taps);
    SLLM_REQUIRE(num_prefill_tokens >= 0 && num_prefill_tokens <= num_tokens, "short_conv: bad number of prompt rows");
    SLLM_REQUIRE(in_dtype == out_dtype || in_dtype == SLLM_F32, "short_conv: the input is fp32 or of the output's type");
    if (num_tokens == 0) return 0;
    SLLM_REQUIRE(xin && w && tok_seq && tok_pos && out && (taps == 1 || tail), "short_conv: null pointer");
    const cudaStream_t st = (cudaStream_t)stream;
#define SC_LAUNCH(TI, TOKENS, r0, r1)                                                                                          \
    short_conv_kernel<TI, T, TOKENS><<<dim3((unsigned)cdiv((r1) - (r0), TOKENS), (unsigned)cdiv(channels, 128)), 128, 0, st>>>(   \
        (const TI*)xin, xin_stride, (const float*)w, (const float*)bias, (TI*)tail, (const int*)tok_seq,                        \
        (const int*)tok_pos, (T*)out, (int64_t)(r0), (int64_t)(r1), channels, taps, add_input, act_silu,                        \
        (TOKENS == 1 && move_decode_tails && taps > 1) ? 1 : 0)
    // prompt rows in pieces of four channels: three or four taps (what the workers have) take the vector kernel, others a channel per thread,
    // which also starts sooner where there are few entries (4 taps, bf16, us: 300 x 2048 12 against 16, 300 x 4096 16 both, 2048 x 516 16
    // both, 2048 x 2048 31 against 18)
    const bool vec = num_prefill_tokens * channels >= (1 << 20) && (taps == 3 || taps == 4) && channels % 4 == 0 && xin_stride % 4 == 0 &&
                     (((uintptr_t)xin | (uintptr_t)tail | (uintptr_t)out | (uintptr_t)w) & 15) == 0;
    // rows of a tile: the fewer, the more CTAs and the shorter a thread's chain of loads; the more, the fewer rows are read twice (4 taps,
    // bf16, us, 8 / 16 / 32 rows: 2^20 entries 8 / 10 / 14, 4 x 2^20 12.5 / 13.4 / 15.7, 6 x 15.9 / 16.5 / 17.7, 8 x 18.7 / 18.4 / 20.5, 24 x
    // 46 / 44 / 46, 32 x 60 / 58 / 57)
    const int64_t entries = num_prefill_tokens * channels;
#define SC_VEC_TILES(TI, K, ROWS)                                                                                              \
    short_conv_vec_kernel<TI, T, K, ROWS><<<dim3((unsigned)cdiv(num_prefill_tokens, ROWS), (unsigned)cdiv(channels, 512)), 128, 0, st>>>( \
        (const TI*)xin, xin_stride, (const float*)w, (const float*)bias, (const TI*)tail, (const int*)tok_seq, (const int*)tok_pos, \
        (T*)out, num_prefill_tokens, channels, add_input, act_silu)
#define SC_VEC(TI, K)                                                                                                          \
    do {                                                                                                                       \
        if (entries < (7 << 20)) SC_VEC_TILES(TI, K, 8);                                                                       \
        else if (entries < (28 << 20)) SC_VEC_TILES(TI, K, 16);                                                                \
        else SC_VEC_TILES(TI, K, 32);                                                                                          \
    } while (0)
    if (num_prefill_tokens > 0 && vec) {
        if (in_dtype == SLLM_F32) { SLLM_DISPATCH_DTYPE_F32(out_dtype, { if (taps == 3) SC_VEC(float, 3); else SC_VEC(float, 4); }); }
        else { SLLM_DISPATCH_DTYPE_F32(out_dtype, { if (taps == 3) SC_VEC(T, 3); else SC_VEC(T, 4); }); }
        if (check_launch("short_conv (prompt portions)")) return 1;
    } else if (num_prefill_tokens > 0) {
        if (in_dtype == SLLM_F32) { SLLM_DISPATCH_DTYPE_F32(out_dtype, (SC_LAUNCH(float, 16, 0, num_prefill_tokens))); }
        else { SLLM_DISPATCH_DTYPE_F32(out_dtype, (SC_LAUNCH(T, 16, 0, num_prefill_tokens))); }
        if (check_launch("short_conv (prompt portions)")) return 1;
    }
    if (num_tokens > num_prefill_tokens) {
        if (in_dtype == SLLM_F32) { SLLM_DISPATCH_DTYPE_F32(out_dtype, (SC_LAUNCH(float, 1, num_prefill_tokens, num_tokens))); }
        else { SLLM_DISPATCH_DTYPE_F32(out_dtype, (SC_LAUNCH(T, 1, num_prefill_tokens, num_tokens))); }
    }
#undef SC_LAUNCH
#undef SC_VEC
#undef SC_VEC_TILES
    return check_launch("short_conv");
}

int sllm_conv_tail_update(const void* xin, int64_t xin_stride, void* tail, const void* seg_starts, const void* seq_ids,
                          const void* tok_pos, int num_segs, int channels, int taps, sllm_dtype_t dtype, sllm_stream_t stream) {
    SLLM_REQUIRE(num_segs >= 0 && channels > 0 && taps >= 1 && taps <= SC_MAX_TAPS, "conv_tail_update: bad shape");
    if (num_segs == 0 || taps == 1) return 0;
    SLLM_REQUIRE(xin && tail && seg_starts && seq_ids && tok_pos, "conv_tail_update: null pointer");
    const dim3 grid((unsigned)num_segs, (unsigned)cdiv(channels, 128));
    SLLM_DISPATCH_DTYPE_F32(dtype, (conv_tail_update_kernel<T><<<grid, 128, 0, (cudaStream_t)stream>>>(
        (const T*)xin, xin_stride, (T*)tail, (const int*)seg_starts, (const int*)seq_ids, (const int*)tok_pos, channels, taps)));
    return check_launch("conv_tail_update");
}

int sllm_mingru_scan(const void* proj, int64_t proj_stride, void* state, const void* seg_starts, const void* seq_ids,
                     const void* tok_pos, void* out, int num_segs, int num_prefill_segs, int channels, sllm_dtype_t dtype,
                     sllm_stream_t stream) {
    SLLM_REQUIRE(num_segs >= 0 && channels > 0 && proj_stride >= 3 * (int64_t)channels, "mingru_scan: bad shape");
    SLLM_REQUIRE(num_prefill_segs >= 0 && num_prefill_segs <= num_segs, "mingru_scan: bad number of prompt segments");
    if (num_segs == 0) return 0;
    SLLM_REQUIRE(proj && state && seg_starts && seq_ids && tok_pos && out, "mingru_scan: null pointer");
    if (num_prefill_segs > 0) {
        const dim3 grid((unsigned)num_prefill_segs, (unsigned)cdiv(channels, 32));
        SLLM_DISPATCH_DTYPE_F32(dtype, (mingru_scan_tiled_kernel<T><<<grid, 256, 0, (cudaStream_t)stream>>>(
            (const T*)proj, proj_stride, (float*)state, (const int*)seg_starts, (const int*)seq_ids, (const int*)tok_pos, (T*)out,
            channels)));
        if (check_launch("mingru_scan (prompt portions)")) return 1;
    }
    if (num_segs > num_prefill_segs) {
        const dim3 grid((unsigned)(num_segs - num_prefill_segs), (unsigned)cdiv(channels, 128));
        SLLM_DISPATCH_DTYPE_F32(dtype, (mingru_scan_kernel<T><<<grid, 128, 0, (cudaStream_t)stream>>>(
            (const T*)proj, proj_stride, (float*)state, (const int*)seg_starts + num_prefill_segs,
            (const int*)seq_ids + num_prefill_segs, (const int*)tok_pos, (T*)out, channels)));
    }
    return check_launch("mingru_scan");
}

int sllm_selective_scan(const void* x, int64_t x_stride, const void* dt, int64_t dt_stride, int dt_f32, const void* dt_bias,
                        const void* A, const void* bc, int64_t bc_stride, int b_off, int c_off, const void* D, const void* z,
                        int64_t z_stride, void* state, const void* seg_starts, const void* seq_ids, const void* tok_pos, void* out,
                        int num_segs, int num_prefill_segs, int channels, int states, sllm_dtype_t dtype, sllm_stream_t stream) {
    return sllm_selective_scan_rows(x, x_stride, dt, dt_stride, dt_f32, dt_bias, A, bc, bc_stride, b_off, c_off, D, z, z_stride, state, seg_starts,
                                    seq_ids, tok_pos, out, -1, num_segs, num_prefill_segs, channels, states, dtype, stream);
}

int sllm_selective_scan_rows(const void* x, int64_t x_stride, const void* dt, int64_t dt_stride, int dt_f32, const void* dt_bias,
                             const void* A, const void* bc, int64_t bc_stride, int b_off, int c_off, const void* D, const void* z,
                             int64_t z_stride, void* state, const void* seg_starts, const void* seq_ids, const void* tok_pos, void* out,
                             int64_t num_tokens, int num_segs, int num_prefill_segs, int channels, int states, sllm_dtype_t dtype,
                             sllm_stream_t stream) {
    SLLM_REQUIRE(num_prefill_segs >= 0 && num_prefill_segs <= num_segs, "selective_scan: bad number of prompt segments");
    SLLM_REQUIRE(num_segs >= 0 && channels > 0 && states > 0 && states <= 32 * SS_R, "selective_scan: 1 <= states <= %d (got %d)",
                 32 * SS_R, states);
    if (num_segs == 0) return 0;
    const int64_t num_prefill_tokens = num_tokens - (num_segs - num_prefill_segs);         // (used where num_tokens >= 0)
    SLLM_REQUIRE(x && dt && dt_bias && A && bc && D && z && state && seg_starts && seq_ids && tok_pos && out,
                 "selective_scan: null pointer");
    int ns_plain = 0;                                  // lanes per channel (log2): the fewest that hold all states
    while ((SS_R << ns_plain) < states) ns_plain++;
    int ns_tiled = ns_plain, sms = 0;
    if (num_prefill_segs > 0) {
        // prompt portions walk their tokens one after the other: with few (segment, channel) pairs more lanes per channel (fewer
        // states per thread) put more warps on the SMs, but not below four states a lane where these are read and multiplied together, four
        // tokens at a time, which takes 16 states or more (512 tokens, 16 states, us: 162 with one state a lane, 68 with four; 24: 174 and
        // 167; 32: 193 and 113; 64: 248 and 134), or where one state a lane would be more than eight warps an SM (8 states: 64 to
        // 4096 channels 156 - 170 and 168, f32 152 - 168 and 195; 8192 channels 215 and 168, f32 211 and 195; 4 states 162 and 287)
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, current_device());
        const int64_t pairs = (int64_t)num_prefill_segs * channels, few = 8 * (int64_t)sms;
        const bool fours = (states & 3) == 0 && (states >= 16 || (states >= 8 && pairs * states / 32 > few));
        while (ns_tiled < 5 && (2 << ns_tiled) <= states && (pairs << ns_tiled) / 32 < few && !(fours && (states >> ns_tiled) <= 4)) ns_tiled++;
    }
    int tt = SS_ITEMS << ns_tiled;                     // tt * (128 >> ns_tiled) = 128 SS_ITEMS entries per staged array ...
    if (tt > 32) tt = 32;
    while (tt > 1 && (size_t)2 * tt * states * sizeof(float) > 24 * 1024) tt >>= 1;                    // ... and B / C rows within 24 KB
    const size_t smem = ((size_t)4 * tt * (128 >> ns_tiled) + (size_t)2 * tt * states) * sizeof(float);   // <= 40 KB
#define SS_GRID(NSEG, NSL) dim3((unsigned)(NSEG), (unsigned)cdiv(channels, 128 >> (NSL))), 128
#define SS_ARGS(TD, SEG0, NSL)                                                                                                 \
    (const T*)x, x_stride, (const TD*)dt, dt_stride, (const float*)dt_bias, (const float*)A, (const T*)bc, bc_stride, b_off,     \
        c_off, (const float*)D, (const T*)z, z_stride, (float*)state, (const int*)seg_starts + (SEG0),                          \
        (const int*)seq_ids + (SEG0), (const int*)tok_pos, (T*)out, channels, states, (NSL)
    const cudaStream_t st = (cudaStream_t)stream;
    if (num_prefill_segs > 0) {
        const int dv = dt_f32 ? 4 : 8;
        const bool vec = dtype != SLLM_F32 && states % 8 == 0 && channels % 8 == 0 && ns_tiled <= 4 && x_stride % 8 == 0 && z_stride % 8 == 0 &&
                         bc_stride % 8 == 0 && b_off % 8 == 0 && c_off % 8 == 0 && dt_stride % dv == 0 &&
                         (((uintptr_t)x | (uintptr_t)dt | (uintptr_t)z | (uintptr_t)bc | (uintptr_t)out) & 15) == 0;
#define SS_TILED(TT, TD, ...) selective_scan_tiled_kernel<TT, TD, __VA_ARGS__><<<SS_GRID(num_prefill_segs, ns_tiled), smem, st>>>(SS_ARGS(TD, 0, ns_tiled), tt)
        // Portions that fill one tile of the kernel for 16 states in part leave its stagers idle, and it holds two or three CTAs on an SM where
        // the tiled one holds eight: many short portions (on the average) stay with that one.  Tiled / own kernel, us: 64 x 8 tokens, 4096
        // channels 28 / 36, 64 x 16, 8192 channels 76 / 104, 8 x 16, 4096 channels 8.1 / 8.2, 32 x 40 41.0 / 43.1; but 4 x 16 5.2 / 4.8, 8 x 1
        // 5.8 / 4.7, 32 x 64 61.1 / 60.9.
        const int64_t pairs = (int64_t)num_prefill_segs * channels, mean = num_prefill_tokens / num_prefill_segs;
        const bool brief = num_tokens >= 0 && ((mean <= 48 && pairs > 600 * (int64_t)sms) || (mean >= 8 && mean <= 24 && pairs > 140 * (int64_t)sms));
        const bool n16 = vec && dt_f32 && states == 16, own = n16 && (((uintptr_t)A | (uintptr_t)state) & 15) == 0;
        if (n16 && ns_tiled == 1 && (brief || !own)) { SLLM_DISPATCH_DTYPE(dtype, (SS_TILED(T, float, true, true))); }
        else if (own) {
            // one channel per lane while all CTAs are on the SMs at once, three each (us, one / two channels: 2 x 777 tokens, 4096 channels
            // 65 / -, 2 x 777, 8192 channels 124 / 100, 3 x 2048, 4096 channels 217 / 248, 4 x 2048, 4096 channels 315 / 247)
            const bool two = (int64_t)num_prefill_segs * cdiv(channels, 32) > 3 * (int64_t)sms;
#define SP_LAUNCH(CPL) do {                                                                                                     \
            static unsigned long long attr_mask = 0;                                                                            \
            auto kern = selective_scan16_kernel<T, CPL>;                                                                        \
            if (first_use_on_this_device(attr_mask)) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SpSmem<CPL>)); \
            kern<<<dim3((unsigned)num_prefill_segs, (unsigned)cdiv(channels, 32 * (CPL))), 128 + 128 * (CPL), sizeof(SpSmem<CPL>), st>>>(     \
                (const T*)x, x_stride, (const float*)dt, dt_stride, (const float*)dt_bias, (const float*)A, (const T*)bc, bc_stride, b_off, c_off, \
                (const float*)D, (const T*)z, z_stride, (float*)state, (const int*)seg_starts, (const int*)seq_ids, (const int*)tok_pos, (T*)out, channels); \
        } while (0)
            SLLM_DISPATCH_DTYPE(dtype, { if (two) SP_LAUNCH(2); else SP_LAUNCH(1); });
#undef SP_LAUNCH
        } else if (vec) {
            if (dt_f32) { SLLM_DISPATCH_DTYPE(dtype, (SS_TILED(T, float, true))); }
            else { SLLM_DISPATCH_DTYPE(dtype, (SS_TILED(T, T, true))); }
        } else if (dt_f32) { SLLM_DISPATCH_DTYPE_F32(dtype, (SS_TILED(T, float, false))); }
        else { SLLM_DISPATCH_DTYPE_F32(dtype, (SS_TILED(T, T, false))); }
#undef SS_TILED
        if (check_launch("selective_scan (prompt portions)")) return 1;
    }
    if (num_segs > num_prefill_segs) {
        const int rest = num_segs - num_prefill_segs;
        if (dt_f32) {
            SLLM_DISPATCH_DTYPE_F32(dtype, (selective_scan_kernel<T, float><<<SS_GRID(rest, ns_plain), 0, st>>>(
                SS_ARGS(float, num_prefill_segs, ns_plain))));
        } else {
            SLLM_DISPATCH_DTYPE_F32(dtype, (selective_scan_kernel<T, T><<<SS_GRID(rest, ns_plain), 0, st>>>(
                SS_ARGS(T, num_prefill_segs, ns_plain))));
        }
    }
#undef SS_ARGS
#undef SS_GRID
    return check_launch("selective_scan");
}

}  // extern "C"
