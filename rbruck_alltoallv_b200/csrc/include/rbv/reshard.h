/* Sequence <-> head re-sharding of sequence-parallel attention for a communicator whose ranks one process hosts.
 * The reference has no attention code; this is its uniform all-to-all with the pack / unpack folded in. */
#ifndef RBV_RESHARD_H_
#define RBV_RESHARD_H_

#include "rbv/rbruckv.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Rank r's sequence-side array is [seq][P][piece_bytes] (its slice of the sequence, all heads; one piece is the heads
 * of one rank), rank q's head-side array is [P * seq][piece_bytes] (the whole sequence, its heads):
 *   head_side[q][r * seq + s] = seq_side[r][s][q]        to_head != 0
 *   seq_side[r][s][q] = head_side[q][r * seq + s]        to_head == 0
 * in one kernel.  The pointer arrays (P entries each) are host arrays of device addresses; the two sides must not
 * overlap.  One process hosting all P <= 64 ranks.  Returns 0 or a CUDA error code. */
int rbv_reshard_heads(rbv_ctx_t ctx, const void* const* seq_side, const void* const* head_side, long long seq,
                      long long piece_bytes, int to_head, void* cuda_stream);

#ifdef __cplusplus
}
#endif
#endif
