// Block compression on strided inputs and outputs (see phi_mlp.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nsa_b200.h"

namespace nsa {

// Scratch and saved sizes as for nsa_cmp_phi_fwd with `arows` tokens, the rows of W1 K that are formed per plane: T, or where
// phi_pool_bwd_fused_ok more, the keys' rows being zero there (T no multiple of 8 lets the products choose a slower kernel).  v_cmp planes and k_cmp rows are nbp apart.
// kc: scratch of BG * dk * (next power of two of the blocks) floats, or null (see phi_mlp.cu).
int cmp_phi_fwd_strided(const void* k, int64_t k_ld, int64_t k_plane, const void* v, const int64_t* vs, const float* pos_embed,
                        const float* w1, const float* b1, const float* w2, const float* b2, float* k_cmp, void* k_cmp_lp, void* v_cmp,
                        int B, int G, int T, int arows, int dk, int dv, int l, int d, int U, int nbp, float* kc, int dtype, void* saved,
                        size_t saved_bytes, void* workspace, size_t workspace_bytes, cudaStream_t st);
int cmp_phi_bwd_ld(const void* k, int64_t k_ld, const float* pos_embed, const float* w1, const float* w2, const void* dk_cmp,
                   const void* dv_cmp, const void* saved, size_t saved_bytes, void* dk_out, void* dv_out, float* dpos, float* dw1, float* db1,
                   float* dw2, float* db2, int B, int G, int T, int arows, int dk, int dv, int l, int d, int U, int nbp, int dtype, void* workspace,
                   size_t workspace_bytes, cudaStream_t st);

// Blocks nb - nb_new .. nb - 1 of a key/value cache from its streams k, v [B,G,..,cap] into its compressed keys and values
// (incremental.cu).
size_t compress_blocks_workspace_bytes(const nsa_decode_desc& d, int dtype);
int compress_blocks(const nsa_decode_desc& d, const void* k, const void* v, int dtype, int param_dtype, void* workspace, cudaStream_t st);

// Pooling backward for l = 32, d = 16 in one pass: da in the I/O type (planes of a and da arows rows apart), dv_out += dv, dc_part [phi_pool_bwd_parts() * BG, l, U].
bool phi_pool_bwd_fused_ok(int l, int d);
int phi_pool_bwd_parts(int BG, int T);
template <typename T>
int phi_pool_bwd_fused(const float* a, const float* c, const float* dhbar, const float* dv_cmp, T* da, float* dc_part, T* dv_out, int BG, int Tn,
                       int arows, int U, int dv, int nb, int nbp, cudaStream_t st);

}  // namespace nsa
