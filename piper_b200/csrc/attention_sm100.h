// Host-side launchers of the causal GQA flash-attention kernels
// (attention_sm100.cu).  qkv is the packed bf16 projection
// [B*S, (Hq + 2*Hkv) * hd] with rotary embedding already applied; S must be
// a multiple of 128 and hd 64 or 128.  Return codes: 0 ok, -1 unsupported
// shape, -2 kernel attribute set-up failed, -3 launch error, >0 CUresult of
// a tensor-map encode.
#pragma once
#include <cuda_runtime.h>

namespace piper {

// out [B*S, Hq*hd] bf16, lse [B, Hq, S] fp32 (natural log).
int attn_fwd(const void* qkv, void* out, float* lse, int B, int S, int Hq, int Hkv, int hd,
             float softmax_scale, int num_sms, int* status, cudaStream_t st);

// Query tiles (1 or 2) that a CTA of attn_fwd works on.
int attn_tiles_per_cta(int B, int S, int Hq, int num_sms);

// d_qkv has the layout of qkv and is fully overwritten.  delta is scratch of
// B*Hq*S floats provided by the caller, scratch attn_bwd_scratch() more or null (dK/dV CTAs are not split then).
int attn_bwd(const void* qkv, const void* out, const void* d_out, const float* lse, float* delta, float* scratch,
             void* d_qkv, int B, int S, int Hq, int Hkv, int hd, float softmax_scale, int num_sms,
             int* status, cudaStream_t st);

// CTAs that share the query heads of a key block in attn_bwd, and the floats of scratch that they exchange sums in.
int attn_bwd_parts(int B, int S, int Hq, int Hkv, int num_sms);
long long attn_bwd_scratch(int B, int S, int Hq, int Hkv, int hd, int num_sms);

}  // namespace piper
