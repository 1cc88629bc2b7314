// Backward of <gO, O> + <gtO, tO> for bf16 / fp16 on tcgen05 tensor cores: which requests the tcgen05 kernels take,
// and which of them.
//   head dimension 64 : bwd_tc5_fused64.cu (one pass; needs a buffer for dQ; index masks, boolean masks
//                       without tile bitmaps, bias) or bwd_tc5_d64.cu (two launches; every mask kind, steps
//                       over dead tiles)
//   head dimension 32 : on half-filled tiles, bwd_tc5_fused64.cu with a workspace for dQ's shares (not key padding, nor with
//                       tile bitmaps), else bwd_tc5_d64.cu
//   head dimension 128: bwd_tc5_pipe128.cu (two launches; every mask kind)
#include "tc5_common.cuh"

namespace jvpfa {

bool bwd_tc5_eligible(const jvpfa_bwd_args& a) {
  if (a.dtype != JVPFA_BF16 && a.dtype != JVPFA_FP16) return false;
  if (!tc5_head_dim(a.D, a.L)) return false;
  const int k = a.mask.kind;
  if (k == JVPFA_MASK_NONE || k == JVPFA_MASK_CAUSAL || k == JVPFA_MASK_KVLEN) return true;
  return (k == JVPFA_MASK_BOOL && a.mask_bits != nullptr && a.mask_bits_t != nullptr) || tc5_mask_layout(a.mask, a.dtype, a.L);
}

int launch_bwd_tc5(const jvpfa_bwd_args& a, cudaStream_t s) {
  if (a.D <= 64) {
    // one pass over the score tiles when the caller gave the dQ accumulation buffer (bwd_tc5_fused64.cu)
    // (for dQ alone the own-queries launch of the two forms 7 of the 10 products of that pass)
    if (bwd_tc5_fused64_eligible(a) && !(a.flags & JVPFA_SKIP_DKDV)) return launch_bwd_tc5_fused64(a, s);
    return launch_bwd_tc5_d64(a, s);  // two pipelined launches (bwd_tc5_d64.cu)
  }
  if (bwd_tc5_pipe128_eligible(a)) return launch_bwd_tc5_pipe128(a, s);  // head dimension 128 (bwd_tc5_pipe128.cu)
  return JVPFA_ERR_UNSUPPORTED;
}

}  // namespace jvpfa
