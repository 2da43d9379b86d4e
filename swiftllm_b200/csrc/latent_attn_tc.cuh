// What latent_attn.cu hands to the tcgen05 kernel of latent_attn_tc.cu.
#pragma once
#include "common.cuh"

namespace sllm {

struct LatentTc {
    const void* q_lat; int64_t ql_st, ql_sh;
    const void* q_rot; int64_t qr_st, qr_sh;
    const float* cosb; const float* sinb;
    const void* gate; int64_t gate_st;
    const void* cache;
    int n_slots, slot, block_size;
    const int* block_table; int max_blocks_per_seq;
    const int* tok_seq; const int* tok_pos;
    void* out; int64_t out_st, out_sh;
    int num_tokens, H, r, dr, rot_dims, window;
    float scale;
    const float* sink;
    int nsplit;
    float* partial;
    int qt, hp_log2;                                 // tokens per CTA; heads per token, padded
    int q_vec, rot_vec, out_vec;                     // 16-byte loads of q_lat, of q_rot and its angles / stores of out are aligned
};

// r in whole 64-column chunks, at most 512; the rotated part at most one chunk (its 16-wide steps are what is multiplied)
bool latent_tc_supported(int r, int dr);
// portions: rows are prompt portions, whose neighbouring tokens share key tiles; otherwise one token per CTA.  Sets qt and hp_log2.
// nsplit > 1 leaves [T, H, nsplit, r + 2] in `partial` for latent_attn_combine_kernel.
int launch_latent_attn_tc(LatentTc& p, bool portions, sllm_dtype_t dtype, cudaStream_t stream);

// latent_attn_prompt.cu: prompt rows of 512 + 64 entries in one key split, on launch_latent_attn_tc's grid; -1: a view that has no tensor map
bool latent_prompt_takes(const LatentTc& p, dim3 grid, int num_sms);
int launch_latent_attn_prompt(const LatentTc& p, dim3 grid, sllm_dtype_t dtype, cudaStream_t stream);

}  // namespace sllm
