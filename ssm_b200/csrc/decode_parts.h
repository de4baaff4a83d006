/* What decode steps of more than 16 sequences are made of besides the entry points of ssm_b200.h: products of a few activation rows with
 * weight matrices on the tensor cores, and the window updates of several convolutions in one launch.  Not part of the C
 * interface: called by the PyTorch extension. */
#ifndef SSM_B200_DECODE_PARTS_H_
#define SSM_B200_DECODE_PARTS_H_
#include <stdint.h>

#include "../../include/ssm_b200.h"

#ifdef __cplusplus
extern "C" {
#endif
enum { SSMB_GEMM_MATS = 5, SSMB_GEMM_MAX_ROWS = 256 };
/* out[i][b * ldo[i] + r] = sum_c x[b * ldx + c] w[i][r * k + c] in io_dtype (bf16 / fp16) with fp32 accumulation, for i < mats,
 * b < batch, r < rows[i].  x, w 16-byte aligned, ldx and k multiples of 8 elements.  status: the word that a wait which runs out sets.
 * weights_ahead: the kernel before this one on the stream does not write the weights, so they may be fetched before it ends. */
typedef struct {
  int32_t batch, k, mats, io_dtype;
  int64_t ldx;
  const void* x;
  const void* w[SSMB_GEMM_MATS];
  int32_t rows[SSMB_GEMM_MATS];
  void* out[SSMB_GEMM_MATS];
  int64_t ldo[SSMB_GEMM_MATS];
  int32_t* status;
  int32_t weights_ahead;
  int32_t plan_rows, plan_splits; /* token rows of a CTA (a multiple of 16) and CTAs that share its columns (1, 2, 4, 8); 0: chosen */
  int32_t reserved0;
} ssmb_rows_gemm_args;
int ssmb_rows_gemm_supported(int32_t batch, int32_t k, int64_t ldx, int32_t io_dtype);
int ssmb_rows_gemm(const ssmb_rows_gemm_args* args, void* stream);
/* ssm_dw_causal_conv_update for up to three windows of the same batch, width, types and activation */
int ssmb_conv_update_many(const ssm_conv_update_args* args, int32_t n, void* stream);
#ifdef __cplusplus
}
#endif
#endif
