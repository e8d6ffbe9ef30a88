// The arguments of a weight-streaming product, as one block that the caller packs: passed one by one, the forty of them took longer
// to convert than the rest of a call (a feed-forward of 4 tokens, 2 launches: 35 us, 28 packed).
#pragma once

struct SkinnyCall {
    const void* w; const void* act; const void* x; const void* delta; const void* norm_w; void* x_out; const void* rows;
    void* out_f32; void* out_bf16; const void* cos_t; const void* sin_t; void* q_out; void* k_cache; void* v_cache;
    const void* positions; const void* token_req; const void* req_slot; const void* block_table; void* stream;
    double eps, out_mult, gate_limit;
    int n, k, norm_w_dtype, m, epilogue, inter, rot_half, interleaved, table_width, page_size, hq, hkv, dim, accumulate, gate_act;
};
