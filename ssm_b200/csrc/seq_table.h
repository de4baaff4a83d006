/* The table of packed sequences that ssm_ssd_args.seq_table describes, formed on the device.  Not part of the C interface: called by the
 * PyTorch extension. */
#ifndef SSM_B200_SEQ_TABLE_H_
#define SSM_B200_SEQ_TABLE_H_
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif
/* cu: num_seqs + 1 boundaries on the device, int64 (wide) or int32.  table: 2 * num_chunks + num_seqs + 1 words; num_chunks is at least what
 * the sequences need (len / chunk + num_seqs always is); chunks beyond are empty.  Boundaries that do not rise from 0 to len give a
 * table that stays inside the tensors; it is the caller who checks them. */
int ssmb_seq_table(const void* cu, int32_t wide, int32_t num_seqs, int32_t len, int32_t num_chunks, int32_t* table, void* stream);
#ifdef __cplusplus
}
#endif
#endif
