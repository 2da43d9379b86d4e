// Prompt portions of the gated delta rule (head_decay.cuh, DELTA) for 16-bit q, k, v: CHUNKS of 32 tokens on the tensor cores, the state
// in fp32 registers.  With S the state at the chunk's start, D(l, j) the product of the decays of tokens l + 1 .. j, D(j) that of all up to j:
//     rhs_j = beta_j (v_j - D(j) S^T k_j),    u = (I + A)^-1 rhs,  A[j][l] = beta_j D(l, j) (k_l . k_j) for l < j,
//     o_j = D(j) S^T q_j + sum_{l <= j} D(l, j) (k_l . q_j) u_l,      S <- D(last) S + sum_l D(l, last) k_l u_l^T.
// The columns of a head's state never mix, so a warp OWNS 16 of them for the whole segment: S^T [16 columns x dk] are the accumulators of
// mma.m16n8k16 (64 registers at dk = 128), and accumulators are the left operands of the next product as they lie: S^T against the
// chunk's keys and queries, rhs^T against (I + A)^-1 - I, u^T against the score matrix and, weighted, against the keys.  Owners
// exchange nothing.  Two more warpgroups work ahead of them, chunk by chunk: STAGERS bring keys and queries (as fp16, each row times a
// power of two that brings its norm near 2^14, which keeps every bit of theirs down to 2^-28 of that norm) and make the chunk's two
// 32 x 32 matrices (exact products of 16-bit numbers, decays in fp32); MAKERS turn logits into decays, invert I + A in fp32 and finish the
// last chunk's outputs.
//
// tcgen05 would need S in tensor memory and a way through registers to split it: five dependent passes per chunk of some 500 to 1000
// cycles each, and at 64 chains (4 sequences x 16 heads) only 64 SMs busy.  Here a chain is spread over four to eight warps that never wait for
// one another's numbers.  Bound: the owner's chain of dependent products (4900 of 5500 cycles per chunk; its 228 products take 1824 on the
// tensor cores), with three warps per scheduler at 0.5 instructions per cycle; code beyond what fits the instruction caches costs more
// than it saves, so loops are kept short (all unrolled: 385 us).  Measured on B200, bf16, 4 x 2048 tokens, 16 heads, 128 x 128: 717 -> 255 us
// with the head norm's 25.
//
// Precision: S, rhs, u and both matrices are fp32 numbers; as operands they are two fp16 numbers each (22 bits and a sign), the second
// one times 2^11 and with sums of its own, so that it has fp16's whole range too: with a column's largest entry at 2^13 (by a power of
// two) an entry keeps its 22 bits down to 2^-27 of that one, and nothing is lost above 2^-49 of it.  The product of two second parts (2^-24 of
// theirs) is left out.  Products are summed in fp32, and the chunk's own sums are made from zero and added to the decayed state once.  The
// state's distance to 64 bits after 2048 tokens: 1.20e-7 (token by token in fp32: 1.22e-7); that of state rows 2^20 below the others of their
// columns, written and read by nearly one-hot keys, at most 3.7e-7 of the row (4.1e-7; with one sum for both parts, which is 3 % faster, 1.4e-5,
// and 7e-3 for rows 2^30 below).
// Every factor is a product of decays <= 1, summed as logarithms over its own range: nothing overflows, whatever the decays.
// A column in which something is not finite, although its state was, goes through the rule token by token in fp32, so that rows before
// the one that brought it stay as they are.
#pragma once

#include "head_decay.cuh"
#include "mma_helpers.cuh"
#include "tc_helpers.cuh"

namespace sllm {

constexpr int DC_TOKENS = 32;
constexpr int DC_GROUP = 128;                // threads of the stagers, of the makers: a warpgroup each
constexpr int DC_BUFS = 3;                   // chunks in shared memory: the owners', the inverse in the making, the next
constexpr int dc_owner_warps(int cw) { return cw == 8 ? 8 : 4; }               // whole warpgroups: registers move between them
constexpr int dc_threads(int cw) { return dc_owner_warps(cw) * 32 + 2 * DC_GROUP; }
constexpr int DC_PITCH = 40;                 // entries between rows of the 32 x 32 matrices (no bank conflicts)
constexpr float DC_UP = 16384.f;             // entries of both matrices (at most 1) are kept times 2^14
constexpr float DC_LOW = 2048.f;             // low parts are kept times 2^11: as large as the high ones, they lose nothing below them

// one chunk's staged data
template <int DKP, int COLS> struct alignas(16) DcBuf {
    unsigned char k[DC_TOKENS * DKP * 2], q[DC_TOKENS * DKP * 2];               // fp16, swizzled 16-byte pieces (tile_off)
    __half n_hi[DC_TOKENS * DC_PITCH], n_lo[DC_TOKENS * DC_PITCH];              // [j][l]: (I + A)^-1 - I
    __half p_hi[DC_TOKENS * DC_PITCH], p_lo[DC_TOKENS * DC_PITCH];              // [j][l]: D(l, j) k_l . q_j (unit vectors)
    unsigned short v[DC_TOKENS * (COLS + 8)];                                   // as stored
    float beta[DC_TOKENS], bd[DC_TOKENS], zq[DC_TOKENS], tail[DC_TOKENS];       // beta | beta D(j) fk | D(j) fq | D(l, last) fk
    float fk[DC_TOKENS], fq[DC_TOKENS], g[DC_TOKENS];                           // staged row -> unit vector; a token's decay
    float keep[4];                                                              // D(last)
};
template <int DKP, int COLS> struct alignas(16) DcSmem {
    DcBuf<DKP, COLS> buf[DC_BUFS];
    unsigned char raw[2][DC_TOKENS * DKP * 2];                                  // the next rows of k and q as stored (tile_off)
    float os[2][DC_TOKENS * (COLS + 4)];                                        // read-outs
    float a[2][DC_TOKENS * 36];                                                 // [l][j]: A[j][l]
    float x[DC_TOKENS * DC_TOKENS];                                             // [l][c]: the inverse, row by row
    float y[DC_TOKENS / 2 * DC_TOKENS / 2];                                     // its lower left quarter in the making
    float d[DC_TOKENS * DC_PITCH];                                              // [j][l]: D(l, j), 0 for l > j
    float dj[DC_TOKENS];                                                        // D(j)
};

__device__ __forceinline__ float dc_pow2(int biased) { return __int_as_float(biased << 23); }
// the larger magnitude, NaN above all
__device__ __forceinline__ float dc_top(float top, float x, float y) {
    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(x), "f"(y));
    return top;
}
__device__ __forceinline__ float dc_top4(float top) {                           // over the four lanes of a column
    const float x = __shfl_xor_sync(0xffffffffu, top, 1);
    top = dc_top(top, x, x);
    const float y = __shfl_xor_sync(0xffffffffu, top, 2);
    return dc_top(top, y, y);
}
__device__ __forceinline__ bool dc_finite(float top) { return top < INFINITY; }
// the power of two (and its inverse) that brings a column whose largest entry is `top` to 2^13
__device__ __forceinline__ void dc_scale(float top, float& up, float& down) {
    const int e = (int)(__float_as_uint(top) >> 23);
    const int b = e >= 255 ? 127 : min(267 - e, 253);
    up = dc_pow2(b);
    down = dc_pow2(254 - b);
}
__device__ __forceinline__ uint32_t dc_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
// x, y (times up: below 2^14) as two fp16 numbers each, the second times DC_LOW
__device__ __forceinline__ void dc_split(float2 x, float2 up, uint32_t& hi, uint32_t& lo) {
    const float2 s = tc::mul2(x, up);
    const __half2 h = __floats2half2_rn(s.x, s.y);
    const float2 f = __half22float2(h), l = tc::mul2(tc::add2(s, make_float2(-f.x, -f.y)), make_float2(DC_LOW, DC_LOW));
    hi = dc_bits(h);
    lo = dc_bits(__floats2half2_rn(l.x, l.y));
}
// two accumulator tiles (columns 2 t, 2 t + 1 of each; rows g and g + 8) -> one left operand, rows times up[0], up[1]
__device__ __forceinline__ void dc_operand(const float (&c0)[4], const float (&c1)[4], const float (&up)[2], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
    const float2 u0 = make_float2(up[0], up[0]), u1 = make_float2(up[1], up[1]);
    dc_split(make_float2(c0[0], c0[1]), u0, hi[0], lo[0]);
    dc_split(make_float2(c0[2], c0[3]), u1, hi[1], lo[1]);
    dc_split(make_float2(c1[0], c1[1]), u0, hi[2], lo[2]);
    dc_split(make_float2(c1[2], c1[3]), u1, hi[3], lo[3]);
}
__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t* b) { mma_16816<__half>(d, a, b[0], b[1]); }
// the same from zero
__device__ __forceinline__ void dc_mma0(float (&d)[4], const uint32_t (&a)[4], const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

template <typename T> __device__ __forceinline__ float dc_lo(uint32_t w) {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) return __uint_as_float(w << 16);
    else return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu)));
}
template <typename T> __device__ __forceinline__ float dc_hi(uint32_t w) {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) return __uint_as_float(w & 0xffff0000u);
    else return __half2float(__ushort_as_half((unsigned short)(w >> 16)));
}

// grid (segments, heads, ceil(dv / (16 CW))), dc_threads(CW) threads
template <typename T, int DKP, int CW>
__global__ void __launch_bounds__(dc_threads(CW), 1) delta_chunk_kernel(const HeadDecayArgs p) {
    constexpr int COLS = 16 * CW, KS = DKP / 16, OW = dc_owner_warps(CW), ALL = CW * 32 + 2 * DC_GROUP, VP = COLS + 8, OP = COLS + 4;
    constexpr int ALL_BAR = 0, STAGE_BAR = 1, MAKE_BAR = 2, DECAY_BAR = 3;       // named barriers
    using Buf = DcBuf<DKP, COLS>;
    extern __shared__ __align__(16) unsigned char dc_smem[];
    DcSmem<DKP, COLS>& sm = *reinterpret_cast<DcSmem<DKP, COLS>*>(dc_smem);
    const int h = blockIdx.y, b = blockIdx.x;
    const int t0 = p.seg_starts[b], n = p.seg_starts[b + 1] - t0;
    if (n <= 0) return;
    const int seq = p.seq_ids[b], dk = p.dk, dv = p.dv, kvh = h / (p.H / p.G), cta_col = blockIdx.z * COLS;
    const bool whole = COLS == 128 && gridDim.z == 1;                            // the CTA owns the head
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (warp >= OW + 4) {
        // ================ makers: gates and decays two chunks ahead of the owners, the inverse one ahead, outputs one behind
        if constexpr (CW == 8) tc::reg_dec<80>();
        else tc::reg_dec<112>();
        const int mw = warp - OW - 4;
        const float pa = p.pa[h], pb = p.pb[h];
        float za = 0.f, zb = 0.f;
        auto fetch = [&](int i0) {                                               // logits: lane = token
            const int64_t row = t0 + min(i0 + lane, n - 1);
            za = p.ga[row * p.ga_stride + h];
            zb = p.gb[row * p.gb_stride + h];
        };
        auto decays = [&](int i0) {                                              // every warp the sums, eight j each
            Buf& B = sm.buf[i0 / DC_TOKENS % DC_BUFS];
            float a = 0.f, beta = 0.f;                                           // past the end: no decay, nothing written
            if (i0 + lane < n) hd_gates<true>(za, zb, pa, pb, 1.f, a, beta);
            if (i0 + DC_TOKENS < n) fetch(i0 + DC_TOKENS);
            // Logarithms are summed from the chunk's start as pairs of fp32 numbers, so that a range's sum is a difference; below -150 (a
            // decay is 0 from -104 on) they are cut off, so that it is one of finite numbers.
            float hi = a < -150.f ? -150.f : a, lo = 0.f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float x = __shfl_up_sync(0xffffffffu, hi, o), y = __shfl_up_sync(0xffffffffu, lo, o);
                if (lane >= o) {                                                 // Knuth's exact sum of two numbers
                    const float s = __fadd_rn(hi, x), z = __fsub_rn(s, hi);
                    lo = __fadd_rn(__fadd_rn(lo, y), __fadd_rn(__fsub_rn(hi, __fsub_rn(s, z)), __fsub_rn(x, z)));
                    hi = s;
                }
            }
            if (mw == 0) {
                const float dj = expf(hi + lo);
                B.beta[lane] = beta; B.g[lane] = expf(a); sm.dj[lane] = dj;
                if (lane == DC_TOKENS - 1) B.keep[0] = dj;
            }
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const int j = 8 * mw + e;
                const float D = expf((__shfl_sync(0xffffffffu, hi, j) - hi) + (__shfl_sync(0xffffffffu, lo, j) - lo));
                sm.d[j * DC_PITCH + lane] = lane <= j ? D : 0.f;
            }
            tc::named_bar_arrive(DECAY_BAR, 2 * DC_GROUP);
        };
        // (I + A)^-1 - I.  Its two diagonal quarters by columns, forward substitution in blocks of eight rows: lane c column c
        auto quarters = [&](int i0) {
            Buf& B = sm.buf[i0 / DC_TOKENS % DC_BUFS];
            const int q0 = lane & 16;                                            // the quarter's first row and column
            const float* a = sm.a[i0 / DC_TOKENS & 1] + q0 * 36 + q0;
#pragma unroll 1
            for (int j0 = 0; j0 < 16; j0 += 8) {
                float x[8], ar[8];
#pragma unroll
                for (int e = 0; e < 8; e++) x[e] = q0 + j0 + e == lane ? 1.f : 0.f;
#pragma unroll 4
                for (int l = 0; l < j0; l++) {
                    hd_row(a + l * 36 + j0, ar);
                    const float y = sm.x[(q0 + l) * DC_TOKENS + lane];
#pragma unroll
                    for (int e = 0; e < 8; e++) x[e] = fmaf(-ar[e], y, x[e]);
                }
#pragma unroll
                for (int l = 0; l < 7; l++) {
                    hd_row(a + (j0 + l) * 36 + j0, ar);
#pragma unroll
                    for (int e = l + 1; e < 8; e++) x[e] = fmaf(-ar[e], x[l], x[e]);
                }
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int j = q0 + j0 + e;
                    sm.x[j * DC_TOKENS + lane] = x[e];
                    const float y = j > lane ? x[e] * DC_UP : 0.f;
                    const __half hi = __float2half_rn(y);
                    B.n_hi[j * DC_PITCH + lane] = hi;
                    B.n_lo[j * DC_PITCH + lane] = __float2half_rn((y - __half2float(hi)) * DC_LOW);
                }
            }
        };
        // the lower left quarter: -(lower right) (A's lower left) (upper left); two columns of one row per lane
        auto corner = [&](int i0) {
            Buf& B = sm.buf[i0 / DC_TOKENS % DC_BUFS];
            const float* a = sm.a[i0 / DC_TOKENS & 1];
            const int r = 4 * mw + (lane >> 3), c = 2 * (lane & 7);
            float2 y = make_float2(0.f, 0.f);
#pragma unroll
            for (int l = 0; l < 16; l++) {
                const float f = a[l * 36 + 16 + r];
                y = tc::fma2(make_float2(f, f), *reinterpret_cast<const float2*>(&sm.x[l * DC_TOKENS + c]), y);
            }
            *reinterpret_cast<float2*>(&sm.y[r * 16 + c]) = y;
            hd_barrier<DC_GROUP>(MAKE_BAR);
            y = make_float2(0.f, 0.f);
#pragma unroll
            for (int l = 0; l < 16; l++) {
                const float f = -sm.x[(16 + r) * DC_TOKENS + 16 + l];
                y = tc::fma2(make_float2(f, f), *reinterpret_cast<const float2*>(&sm.y[l * 16 + c]), y);
            }
            uint32_t hi, lo;
            dc_split(y, make_float2(DC_UP, DC_UP), hi, lo);
            *reinterpret_cast<uint32_t*>(&B.n_hi[(16 + r) * DC_PITCH + c]) = hi;
            *reinterpret_cast<uint32_t*>(&B.n_lo[(16 + r) * DC_PITCH + c]) = lo;
        };
        // the chunk's read-outs: norm, gate and store where the CTA owns the head, else to the head norm's launch
        auto finish = [&](int i0, int w, int warps) {                            // warp w of that many
            const int nt = min(DC_TOKENS, n - i0);
            const float* os = sm.os[i0 / DC_TOKENS & 1];
            if (!whole) {
                constexpr int LR = COLS / 4, ROWS = 32 / LR;                     // lanes of a row, rows at a time
                const int c = 4 * (lane % LR);
                float* raw = p.o_raw + ((int64_t)(t0 + i0) * p.H + h) * dv + cta_col;
#pragma unroll 2
                for (int j = w * ROWS + lane / LR; j < nt; j += warps * ROWS) {
                    const float4 x = *reinterpret_cast<const float4*>(os + j * OP + c);
                    if (cta_col + c < dv) *reinterpret_cast<float4*>(raw + (int64_t)j * p.H * dv + c) = x;
                }
            } else if constexpr (COLS == 128) {
                const T* gp = (const T*)p.gate + (int64_t)h * dv;
                float nw[4];
#pragma unroll
                for (int c = 0; c < 4; c++) nw[c] = 4 * lane + c < dv ? p.norm_w[h * p.norm_step + 4 * lane + c] : 0.f;
#pragma unroll 1
                for (int j0 = 4 * w; j0 < nt; j0 += 4 * warps) {
                    HdRaw<T, 4> gate[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int j = j0 + u;
                        gate[u].zero();
                        if (j < nt) gate[u].load(gp + (int64_t)(t0 + i0 + j) * p.gate_stride, 4 * lane, dv, p.vec);
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int j = j0 + u;
                        if (j >= nt) break;
                        const float4 x = *reinterpret_cast<const float4*>(os + j * OP + 4 * lane);      // columns past dv are zero
                        float o[4] = {x.x, x.y, x.z, x.w};
                        const float f = rsqrtf(warp_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w) / (float)dv + p.eps);
#pragma unroll
                        for (int c = 0; c < 4; c++) o[c] *= f * nw[c] * hd_act<true>(gate[u].get(c));
                        hd_put<T, 4>((T*)p.out + (t0 + i0 + j) * p.out_stride + (int64_t)h * dv, 4 * lane, dv, p.vec, o);
                    }
                }
            }
        };
        fetch(0);
        decays(0);
        hd_barrier<ALL>(ALL_BAR);
        if (DC_TOKENS < n) decays(DC_TOKENS);
        if (mw == 0) quarters(0);
        hd_barrier<DC_GROUP>(MAKE_BAR);
        corner(0);
        hd_barrier<ALL>(ALL_BAR);
        for (int i0 = 0; i0 < n; i0 += DC_TOKENS) {                              // while the owners work on the chunk at i0
            if (i0 + 2 * DC_TOKENS < n) decays(i0 + 2 * DC_TOKENS);
            const bool more = i0 + DC_TOKENS < n;
            if (mw == 0 && more) quarters(i0 + DC_TOKENS);
            if (mw != 0 && i0 > 0) finish(i0 - DC_TOKENS, mw - 1, 3);
            if (more) {
                hd_barrier<DC_GROUP>(MAKE_BAR);
                corner(i0 + DC_TOKENS);
            }
            hd_barrier<ALL>(ALL_BAR);
        }
        finish((n - 1) / DC_TOKENS * DC_TOKENS, mw, 4);
        return;
    }
    if (warp >= OW) {
        // ================ stagers, two chunks ahead of the owners: a token's row is staged by four neighbouring lanes, eight tokens by a warp
        if constexpr (CW == 8) tc::reg_dec<80>();
        else tc::reg_dec<144>();
        constexpr int KP = DKP / 32, NV = COLS >= 32 ? COLS / 32 : 1;          // 16-byte pieces of a row of k, v per lane
        const int hw = warp - OW, tok = 8 * hw + g;
        const T* vp = (const T*)p.v + (int64_t)h * dv + cta_col;
        auto fetch = [&](int i0) {                                               // rows of k and q, read again by the lane that brings them
            const bool live = i0 + tok < n;
            const int64_t row = t0 + (live ? i0 + tok : 0);
            const T* kp = (const T*)p.k + (int64_t)kvh * dk + row * p.k_stride;
            const T* qp = (const T*)p.q + (int64_t)kvh * dk + row * p.q_stride;
#pragma unroll
            for (int i = 0; i < KP; i++) {
                const int e = 8 * (t + 4 * i), size = live && e < dk ? 16 : 0, at = tile_off<DKP>(tok, t + 4 * i);
                cp_async16(smem_u32(sm.raw[0] + at), size ? kp + e : kp, size);
                cp_async16(smem_u32(sm.raw[1] + at), size ? qp + e : qp, size);
            }
            cp_async_commit();
        };
        auto prepare = [&](int i0) {                                             // the chunk at i0 (fetched before)
            Buf& B = sm.buf[i0 / DC_TOKENS % DC_BUFS];
            float* sa = sm.a[i0 / DC_TOKENS & 1];
            cp_async_wait<0>();
            {
                const bool live = i0 + tok < n;
                const T* row = vp + (int64_t)(t0 + (live ? i0 + tok : 0)) * p.v_stride;
#pragma unroll
                for (int i = 0; i < NV; i++) {
                    const int e = 8 * (t + 4 * i), size = live && cta_col + e < dv ? 16 : 0;
                    if (e < COLS) cp_async16(smem_u32(&B.v[tok * VP + e]), size ? row + e : row, size);
                }
                cp_async_commit();
            }
            // the rows times a power of two, and the factor that makes the staged row a unit vector
#pragma unroll 1
            for (int which = 0; which < 2; which++) {
                unsigned char* tile = which ? B.q : B.k;
                uint32_t w[KP][4];
                float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
                for (int i = 0; i < KP; i++) {
                    const uint4 r = *reinterpret_cast<const uint4*>(sm.raw[which] + tile_off<DKP>(tok, t + 4 * i));
                    w[i][0] = r.x; w[i][1] = r.y; w[i][2] = r.z; w[i][3] = r.w;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const float2 x = make_float2(dc_lo<T>(w[i][c]), dc_hi<T>(w[i][c]));
                        s2 = tc::fma2(x, x, s2);
                    }
                }
                float ss = s2.x + s2.y;
                ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                ss += __shfl_xor_sync(0xffffffffu, ss, 2);
                const int e = (int)((__float_as_uint(ss) >> 23) & 255u);         // a norm of 2^((e - 127) / 2) -> near 2^14
                const int up = e == 255 ? 1 : min(max(127 + 14 - ((e - 127) >> 1), 1), 253);
                const float f = dc_pow2(up);
#pragma unroll
                for (int i = 0; i < KP; i++) {
#pragma unroll
                    for (int c = 0; c < 4; c++) w[i][c] = dc_bits(__floats2half2_rn(dc_lo<T>(w[i][c]) * f, dc_hi<T>(w[i][c]) * f));
                    *reinterpret_cast<uint4*>(tile + tile_off<DKP>(tok, t + 4 * i)) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
                }
                if (t == 0) (which ? B.fq : B.fk)[tok] = rsqrtf(ss + HD_UNIT_EPS) * dc_pow2(254 - up);
            }
            if (i0 + DC_TOKENS < n) fetch(i0 + DC_TOKENS);                       // in flight while this chunk is worked on
            hd_barrier<DC_GROUP>(STAGE_BAR);
            // keys (even warps) and queries (odd ones) against keys: warps 0 and 1 rows 16 .. 31, warps 2 and 3 rows 0 .. 15.  Entries above the
            // diagonal are not read.
            const bool of_q = hw & 1;
            const int m0 = hw < 2 ? 16 : 0;
            float c[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++) c[i][0] = c[i][1] = c[i][2] = c[i][3] = 0.f;
            {
                const uint32_t at = smem_u32(of_q ? B.q : B.k), kt = smem_u32(B.k);
                const int r = (lane & 7) + ((lane >> 4) << 3);
#pragma unroll 2
                for (int ks = 0; ks < KS; ks++) {
                    uint32_t x[4], y[8];
                    ldmatrix_x4(at + tile_off<DKP>(m0 + (lane & 15), 2 * ks + (lane >> 4)), x[0], x[1], x[2], x[3]);
#pragma unroll
                    for (int i = 0; i < 4; i += 2)
                        ldmatrix_x4(kt + tile_off<DKP>(8 * i + r, 2 * ks + ((lane >> 3) & 1)), y[2 * i], y[2 * i + 1], y[2 * i + 2], y[2 * i + 3]);
#pragma unroll
                    for (int i = 0; i < 4; i++) dc_mma(c[i], x, y + 2 * i);
                }
            }
            hd_barrier<2 * DC_GROUP>(DECAY_BAR);                                 // decays are written
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int j = m0 + g + 8 * e;
                const float f = of_q ? B.fq[j] : B.fk[j] * B.beta[j];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int l = 8 * i + 2 * t;
                    const float2 d = *reinterpret_cast<const float2*>(&sm.d[j * DC_PITCH + l]), fk = *reinterpret_cast<const float2*>(&B.fk[l]);
                    const float v0 = c[i][2 * e] * f * fk.x * d.x, v1 = c[i][2 * e + 1] * f * fk.y * d.y;
                    if (of_q) {
                        uint32_t hi, lo;
                        dc_split(make_float2(l <= j ? v0 : 0.f, l + 1 <= j ? v1 : 0.f), make_float2(DC_UP, DC_UP), hi, lo);
                        *reinterpret_cast<uint32_t*>(&B.p_hi[j * DC_PITCH + l]) = hi;
                        *reinterpret_cast<uint32_t*>(&B.p_lo[j * DC_PITCH + l]) = lo;
                    } else {
                        sa[l * 36 + j] = v0;
                        sa[(l + 1) * 36 + j] = v1;
                    }
                }
            }
            if (hw == 1) B.tail[lane] = sm.d[(DC_TOKENS - 1) * DC_PITCH + lane] * B.fk[lane];
            if (hw == 2) B.bd[lane] = B.beta[lane] * sm.dj[lane] * B.fk[lane];
            if (hw == 3) B.zq[lane] = sm.dj[lane] * B.fq[lane];
            if (i0 + DC_TOKENS < n) cp_async_wait<1>();                          // v is there
            else cp_async_wait<0>();
        };
        fetch(0);
        prepare(0);
        hd_barrier<ALL>(ALL_BAR);
        if (DC_TOKENS < n) prepare(DC_TOKENS);
        hd_barrier<ALL>(ALL_BAR);
        for (int i0 = 0; i0 < n; i0 += DC_TOKENS) {                              // while the owners work on the chunk at i0
            if (i0 + 2 * DC_TOKENS < n) prepare(i0 + 2 * DC_TOKENS);
            hd_barrier<ALL>(ALL_BAR);
        }
        return;
    }
    // ================ owners: columns c0 = cta_col + 16 warp + g and c0 + 8 of the state; keys 8 i + 2 t, 8 i + 2 t + 1 (i: the tile)
    if constexpr (CW == 8) tc::reg_inc<176>();
    else tc::reg_inc<240>();
    if (warp >= CW) return;
    const int c0 = 16 * warp + g;
    float* st = p.state + ((int64_t)seq * p.H + h) * dk * dv + cta_col;
    const bool fresh = p.tok_pos[t0] == 0;
    float S[DKP / 8][4];
    float top[2];                                                                // largest |entry| of this lane's part of its two columns
    auto measure = [&]() {
        top[0] = top[1] = 0.f;
#pragma unroll
        for (int i = 0; i < DKP / 8; i++)
#pragma unroll
            for (int r = 0; r < 2; r++) top[r] = dc_top(top[r], S[i][2 * r], S[i][2 * r + 1]);
    };
#pragma unroll
    for (int i = 0; i < DKP / 8; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int d = 8 * i + 2 * t + (e & 1), c = c0 + 8 * (e >> 1);
            S[i][e] = (!fresh && d < dk && cta_col + c < dv) ? st[(int64_t)d * dv + c] : 0.f;
        }
    measure();
    const int r16 = (lane & 7) + ((lane >> 4) << 3), ch2 = (lane >> 3) & 1;      // two tiles of eight rows, two pieces (ldmatrix)
    hd_barrier<ALL>(ALL_BAR);
    hd_barrier<ALL>(ALL_BAR);
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += DC_TOKENS) {
        const Buf& B = sm.buf[i0 / DC_TOKENS % DC_BUFS];
        float* os = sm.os[i0 / DC_TOKENS & 1] + c0;
        const uint32_t kt = smem_u32(B.k), qt = smem_u32(B.q);
        top[0] = dc_top4(top[0]); top[1] = dc_top4(top[1]);
        const bool sound[2] = {dc_finite(top[0]), dc_finite(top[1])};
        float up[2], down[2];
        dc_scale(top[0], up[0], down[0]); dc_scale(top[1], up[1], down[1]);
        // ---- the state against keys (R) and queries (Z)
        float R[4][4], Rl[4][4], Z[4][4], Zl[4][4];
#pragma unroll
        for (int ks = 0; ks < KS; ks++) {
            uint32_t hi[4], lo[4], kb[8], qb[8];
            ldmatrix_x4(kt + tile_off<DKP>(r16, 2 * ks + ch2), kb[0], kb[1], kb[2], kb[3]);
            ldmatrix_x4(kt + tile_off<DKP>(16 + r16, 2 * ks + ch2), kb[4], kb[5], kb[6], kb[7]);
            ldmatrix_x4(qt + tile_off<DKP>(r16, 2 * ks + ch2), qb[0], qb[1], qb[2], qb[3]);
            ldmatrix_x4(qt + tile_off<DKP>(16 + r16, 2 * ks + ch2), qb[4], qb[5], qb[6], qb[7]);
            dc_operand(S[2 * ks], S[2 * ks + 1], up, hi, lo);
            if (ks == 0) {
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma0(Rl[i], lo, kb + 2 * i);
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma0(Zl[i], lo, qb + 2 * i);
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma0(R[i], hi, kb + 2 * i);
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma0(Z[i], hi, qb + 2 * i);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma(Rl[i], lo, kb + 2 * i);
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma(Zl[i], lo, qb + 2 * i);
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma(R[i], hi, kb + 2 * i);
#pragma unroll
                for (int i = 0; i < 4; i++) dc_mma(Z[i], hi, qb + 2 * i);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) Z[i][e] = fmaf(Zl[i][e], 1.f / DC_LOW, Z[i][e]);
        // ---- rhs = beta (v - D(j) S^T k), in R
        float xt[2] = {0.f, 0.f};
        {
            uint32_t vb[8];                                                      // [tile]: columns g and g + 8, tokens 2 t and 2 t + 1
            const uint32_t va = smem_u32(B.v) + (r16 * VP + 16 * warp + 8 * ch2) * 2;
            ldmatrix_x4_trans(va, vb[0], vb[1], vb[2], vb[3]);
            ldmatrix_x4_trans(va + 16 * VP * 2, vb[4], vb[5], vb[6], vb[7]);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 bt = *reinterpret_cast<const float2*>(&B.beta[8 * i + 2 * t]), bd = *reinterpret_cast<const float2*>(&B.bd[8 * i + 2 * t]);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const uint32_t w = vb[2 * i + r];
                    const float x = fmaf(Rl[i][2 * r], 1.f / DC_LOW, R[i][2 * r]) * down[r], y = fmaf(Rl[i][2 * r + 1], 1.f / DC_LOW, R[i][2 * r + 1]) * down[r];
                    R[i][2 * r] = fmaf(-bd.x, x, bt.x * dc_lo<T>(w));
                    R[i][2 * r + 1] = fmaf(-bd.y, y, bt.y * dc_hi<T>(w));
                    xt[r] = dc_top(xt[r], R[i][2 * r], R[i][2 * r + 1]);
                }
            }
        }
        // ---- R through (I + A)^-1: u, then u through the scores: the read-outs' part within the chunk.  Token j's sums are over l <= j.
        bool odd = false;
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) {
            xt[0] = dc_top4(xt[0]); xt[1] = dc_top4(xt[1]);
            odd = odd || (sound[0] && !dc_finite(xt[0])) || (sound[1] && !dc_finite(xt[1]));
            float u2[2], dn[2], E[4][4], El[4][4];
            dc_scale(xt[0], u2[0], dn[0]); dc_scale(xt[1], u2[1], dn[1]);
            dn[0] *= 1.f / DC_UP; dn[1] *= 1.f / DC_UP;
            const uint32_t mh = smem_u32(pass ? B.p_hi : B.n_hi) + (r16 * DC_PITCH + 8 * ch2) * 2;
            constexpr uint32_t LO = DC_TOKENS * DC_PITCH * 2, DOWN = 16 * DC_PITCH * 2, RIGHT = 32;      // bytes to the low part, 16 rows down, 16 columns on
            uint32_t hi[4], lo[4], b0[4], b1[4], l0[4], l1[4];
            ldmatrix_x4(mh, b0[0], b0[1], b0[2], b0[3]);
            ldmatrix_x4(mh + LO, l0[0], l0[1], l0[2], l0[3]);
            ldmatrix_x4(mh + DOWN, b1[0], b1[1], b1[2], b1[3]);
            ldmatrix_x4(mh + LO + DOWN, l1[0], l1[1], l1[2], l1[3]);
            dc_operand(R[0], R[1], u2, hi, lo);
#pragma unroll
            for (int i = 0; i < 2; i++) { dc_mma0(El[i], hi, l0 + 2 * i); dc_mma0(El[2 + i], hi, l1 + 2 * i); }
#pragma unroll
            for (int i = 0; i < 2; i++) { dc_mma(El[i], lo, b0 + 2 * i); dc_mma(El[2 + i], lo, b1 + 2 * i); }
#pragma unroll
            for (int i = 0; i < 2; i++) { dc_mma0(E[i], hi, b0 + 2 * i); dc_mma0(E[2 + i], hi, b1 + 2 * i); }
            ldmatrix_x4(mh + DOWN + RIGHT, b1[0], b1[1], b1[2], b1[3]);
            ldmatrix_x4(mh + LO + DOWN + RIGHT, l1[0], l1[1], l1[2], l1[3]);
            dc_operand(R[2], R[3], u2, hi, lo);
#pragma unroll
            for (int i = 0; i < 2; i++) dc_mma(El[2 + i], hi, l1 + 2 * i);
#pragma unroll
            for (int i = 0; i < 2; i++) dc_mma(El[2 + i], lo, b1 + 2 * i);
#pragma unroll
            for (int i = 0; i < 2; i++) dc_mma(E[2 + i], hi, b1 + 2 * i);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int e = 0; e < 4; e++) E[i][e] = fmaf(El[i][e], 1.f / DC_LOW, E[i][e]);
            if (pass == 0) {
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        R[i][2 * r] = fmaf(E[i][2 * r], dn[r], R[i][2 * r]);
                        R[i][2 * r + 1] = fmaf(E[i][2 * r + 1], dn[r], R[i][2 * r + 1]);
                        xt[r] = dc_top(i ? xt[r] : 0.f, R[i][2 * r], R[i][2 * r + 1]);
                    }
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float2 zq = *reinterpret_cast<const float2*>(&B.zq[8 * i + 2 * t]);
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        os[(8 * i + 2 * t + (e & 1)) * OP + 8 * (e >> 1)] = fmaf(E[i][e], dn[e >> 1], Z[i][e] * down[e >> 1] * (e & 1 ? zq.y : zq.x)) * p.q_scale;
                }
            }
        }
        if (__builtin_expect(__any_sync(0xffffffffu, odd), 0)) {
            // ---- something new is not finite: token by token in fp32
            const int nt = min(DC_TOKENS, n - i0);
#pragma unroll 1
            for (int j = 0; j < nt; j++) {
                auto at = [&](const unsigned char* tile, int i) { return __half22float2(*reinterpret_cast<const __half2*>(tile + tile_off<DKP>(j, i) + 4 * t)); };
                auto column = [&](float x) {
                    x += __shfl_xor_sync(0xffffffffu, x, 1);
                    return x + __shfl_xor_sync(0xffffffffu, x, 2);
                };
                const float decay = B.g[j], fk = B.fk[j], fq = B.fq[j], beta = B.beta[j];
                float u[2] = {0.f, 0.f}, o[2] = {0.f, 0.f};
#pragma unroll
                for (int i = 0; i < DKP / 8; i++) {
                    const float2 k2 = at(B.k, i);
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        S[i][2 * r] *= decay; S[i][2 * r + 1] *= decay;
                        u[r] = fmaf(S[i][2 * r], k2.x * fk, fmaf(S[i][2 * r + 1], k2.y * fk, u[r]));
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; r++) u[r] = beta * (dc_lo<T>(B.v[j * VP + c0 + 8 * r]) - column(u[r]));
#pragma unroll
                for (int i = 0; i < DKP / 8; i++) {
                    const float2 k2 = at(B.k, i), q2 = at(B.q, i);
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        S[i][2 * r] = fmaf(k2.x * fk, u[r], S[i][2 * r]);
                        S[i][2 * r + 1] = fmaf(k2.y * fk, u[r], S[i][2 * r + 1]);
                        o[r] = fmaf(S[i][2 * r], q2.x * fq, fmaf(S[i][2 * r + 1], q2.y * fq, o[r]));
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const float x = column(o[r]) * p.q_scale;
                    if (t == 0) os[j * OP + 8 * r] = x;
                }
            }
            measure();
            hd_barrier<ALL>(ALL_BAR);
            continue;
        }
        // ---- the state moves on: u times D(l, last) against the keys
        uint32_t wh[2][4], wl[2][4];
        float wd[2];
        {
            float wt[2] = {0.f, 0.f}, wu[2];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 tl = *reinterpret_cast<const float2*>(&B.tail[8 * i + 2 * t]);
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    R[i][2 * r] *= tl.x; R[i][2 * r + 1] *= tl.y;
                    wt[r] = dc_top(wt[r], R[i][2 * r], R[i][2 * r + 1]);
                }
            }
            dc_scale(dc_top4(wt[0]), wu[0], wd[0]); dc_scale(dc_top4(wt[1]), wu[1], wd[1]);
            dc_operand(R[0], R[1], wu, wh[0], wl[0]);
            dc_operand(R[2], R[3], wu, wh[1], wl[1]);
        }
        const float2 keep = make_float2(B.keep[0], B.keep[0]);
        top[0] = top[1] = 0.f;
        constexpr int TILES = 4;                                                  // tiles of eight keys at a time
#pragma unroll
        for (int i1 = 0; i1 < DKP / 8; i1 += TILES) {
            float acc[TILES][4], low[TILES][4];
            uint32_t kb[2][2 * TILES];
#pragma unroll
            for (int ks = 0; ks < 2; ks++)
#pragma unroll
                for (int i = 0; i < TILES; i += 2)                               // rows (tokens) 16 ks .. + 15, pieces i1 + i and i1 + i + 1
                    ldmatrix_x4_trans(kt + tile_off<DKP>(16 * ks + (lane & 15), i1 + i + (lane >> 4)), kb[ks][2 * i], kb[ks][2 * i + 1], kb[ks][2 * i + 2], kb[ks][2 * i + 3]);
#pragma unroll
            for (int i = 0; i < TILES; i++) dc_mma0(low[i], wl[0], kb[0] + 2 * i);
#pragma unroll
            for (int i = 0; i < TILES; i++) dc_mma0(acc[i], wh[0], kb[0] + 2 * i);
#pragma unroll
            for (int i = 0; i < TILES; i++) dc_mma(low[i], wl[1], kb[1] + 2 * i);
#pragma unroll
            for (int i = 0; i < TILES; i++) dc_mma(acc[i], wh[1], kb[1] + 2 * i);
#pragma unroll
            for (int i = 0; i < TILES; i++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    float* x = &S[i1 + i][2 * r];
                    const float2 a = tc::fma2(make_float2(low[i][2 * r], low[i][2 * r + 1]), make_float2(1.f / DC_LOW, 1.f / DC_LOW), make_float2(acc[i][2 * r], acc[i][2 * r + 1]));
                    const float2 y = tc::fma2(a, make_float2(wd[r], wd[r]), tc::mul2(make_float2(x[0], x[1]), keep));
                    x[0] = y.x; x[1] = y.y;
                    top[r] = dc_top(top[r], y.x, y.y);
                }
        }
        hd_barrier<ALL>(ALL_BAR);                                                       // the next chunk is prepared, `os` is written
    }
#pragma unroll
    for (int i = 0; i < DKP / 8; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int d = 8 * i + 2 * t + (e & 1), c = c0 + 8 * (e >> 1);
            if (d < dk && cta_col + c < dv) st[(int64_t)d * dv + c] = S[i][e];
        }
}

// ---------------------------------------------------------------- launchers
template <typename T, int DKP, int CW> static int delta_chunk_launch(const HeadDecayArgs& a, cudaStream_t stream) {
    static unsigned long long attr_mask = 0;
    auto kern = delta_chunk_kernel<T, DKP, CW>;
    const size_t smem = sizeof(DcSmem<DKP, 16 * CW>);
    if (first_use_on_this_device(attr_mask)) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int slices = cdiv(a.dv, 16 * CW);
    kern<<<dim3((unsigned)a.num_segs, (unsigned)a.H, (unsigned)slices), dc_threads(CW), smem, stream>>>(a);
    return CW == 8 && slices == 1 ? 1 : 2;
}

template <typename T, int DKP> static int delta_chunk_width(const HeadDecayArgs& a, int cw, cudaStream_t s) {
    if (cw == 8) return delta_chunk_launch<T, DKP, 8>(a, s);
    if (cw == 4) return delta_chunk_launch<T, DKP, 4>(a, s);
    if (cw == 2) return delta_chunk_launch<T, DKP, 2>(a, s);
    return delta_chunk_launch<T, DKP, 1>(a, s);
}

// The narrowest slices of a head that give no SM two CTAs: an SM holds one, and its owners go the faster the fewer they are.
static inline int delta_chunk_slice(const HeadDecayArgs& a, int num_sms) {
    int cw = 1;
    while (cw < 8 && (int64_t)a.num_segs * a.H * cdiv(a.dv, 16 * cw) > num_sms) cw *= 2;
    return cw;
}

// Rows in 16-byte pieces, at most 128 state rows (more do not fit an owner's registers), and portions that are not too short on the average:
// three staged phases and the inverse take 9 us whatever a chunk holds, a batch of eight tokens 2 to 4, and where a batch kernel's CTA owns a
// head (`owned`) there is no launch for the norm.  Batches / chunks, us, 16 heads: 128 x 128, 1 portion of 8 tokens 7.4 / 10.1, 4 x 8 9.8 / 11.1,
// 9 x 8 14.0 / 12.7, 1 x 16 10.1 / 10.5, 4 x 12 12.5 / 11.2; 64 x 128, 9 x 8 9.3 / 9.7, 9 x 12 12.0 / 9.7; 64 x 64, 4 x 16 8.9 / 9.4, 4 x 20
// 10.8 / 9.3, 9 x 24 9.8 / 10.0, 16 x 24 18.2 / 20.4, 16 x 32 22.2 / 20.5; 32 x 32, 1 x 24 8.5 / 8.9, 16 x 32 19.6 / 20.0; 96 x 160, 2 x 8 10.0 / 11.2, 6 x 8
// 17.8 / 23.9, but 3 x 8, whose chunk kernel has 144 CTAs, 14.7 / 11.5.
static inline bool delta_chunk_takes(const HeadDecayArgs& a, sllm_dtype_t dtype, int64_t num_tokens, int num_sms) {
    const int64_t units = (int64_t)a.num_segs * a.H, ctas = units * cdiv(a.dv, 16 * delta_chunk_slice(a, num_sms));
    const bool owned = a.dv <= 32 || 5 * units >= 3 * (int64_t)num_sms, full = 10 * ctas >= 9 * (int64_t)num_sms && ctas <= num_sms;
    int shortest = 9;
    if (a.dv <= 64) shortest = owned ? 25 : 17;
    else if (a.dv > 128 ? full : owned && a.dk > 64) shortest = 1;
    return num_tokens >= (int64_t)shortest * a.num_segs && dtype != SLLM_F32 && a.dk <= 128 && a.dk % 8 == 0 && a.dv % 8 == 0 &&
           ((a.q_stride | a.k_stride | a.v_stride) & 7) == 0 && (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.o_raw) & 15) == 0;
}

// -> 1: the outputs are finished; 2: the read-outs are in o_raw
template <typename T> static int delta_chunk(const HeadDecayArgs& a, int num_sms, cudaStream_t s) {
    const int cw = delta_chunk_slice(a, num_sms);
    return a.dk <= 64 ? delta_chunk_width<T, 64>(a, cw, s) : delta_chunk_width<T, 128>(a, cw, s);
}

}  // namespace sllm
