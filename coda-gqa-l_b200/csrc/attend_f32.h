// Arguments of the shape-generic attention kernels, and the single-precision kernel among them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct AttnParams {
  int B, H, Hkv, Dh, Lbuf, Lq, mask_unused, norm_full;
  float eps, scale_log2;
  const void* q; long long q_bs, q_rs;
  const void* qn; long long qn_bs, qn_rs;
  const float* lam; long long lam_bs, lam_rs;
  const void* kbuf; const void* vbuf; const uint8_t* allowed;
  const void* kblk; long long kb_bs, kb_rs;
  const void* vblk; long long vb_bs, vb_rs;
  const void* norm_w;
  void* out; long long out_bs, out_rs;
};

// True when the register-tiled single-precision kernel covers the call (head_dim, alignment of rows).
bool coda_attend_f32_supported(const AttnParams& p);
int coda_attend_f32(const AttnParams& p, cudaStream_t s);
