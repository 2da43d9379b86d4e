// What window_attn.cu hands to the tcgen05 kernel of window_attn_tc.cu (prompt rows, 16-bit storage); names as there.
#pragma once
#include "common.cuh"

namespace sllm {

struct WindowTc {
    const void* q; int64_t q_st;
    const float* cosb; const float* sinb;
    const void* gate; int64_t gate_st;
    const void* cache;
    int n_slots, slot, block_size;
    const int* block_table; int max_blocks_per_seq;
    const int* tok_seq; const int* tok_pos;
    void* out; int64_t out_st;
    int beside;                                          // CTAs of decoded rows on a stream beside this launch's
    int group_blocks;                                    // set at the launch: blocks of rows a group, where its CTAs keep together
    int num_rows, H, G, dk, dv, rot_dims, window;
    float scale, sink;
    int halves;
    float qk_norm_eps, softcap;
    const float* vcos; const float* vsin;
    float out_scale;
    const float* qnorm_w;
    float prenorm_eps;
    int chunk, vshare, out_f32;
    const float* slopes;
    int keep_first, gate_per_head, shared_kv, krot;
    const float* sinks;
    int row_elems, koff;                             // entries of a cache row; first key entry
    int qt, hqp_log2;                                // tokens per CTA; heads per group, padded to a power of two
    // 16-byte accesses of q / gate / out are aligned; q_fast: of q and its angles, whose pairs are neighbours
    int q_vec, q_fast, gate_vec, out_vec;
};

// what the products can be cut from (see the kernel); everything else takes the mma.sync kernel
bool window_tc_supported(int dk, int dv, int krot, int hq, float scale, const void* cache, int64_t num_rows);
int launch_window_attn_tc(WindowTc& p, sllm_dtype_t dtype, cudaStream_t stream);

}  // namespace sllm
