/* rows_mma.cuh — launch interface of the integer-flavour row kernel of the M > 1 paths (rows_mma.cu): Q4B weight rows
 * times the int8-quantised activations of a few tokens, for the shared expert and the routed experts in one launch. */
#pragma once
#include "common.cuh"

/* The rows of one tensor (or of one per group) and the activations each group multiplies. */
struct SpRowsSeg {
    const uint8_t *codes, *ucodes;                 /* [groups * rows_per_group][in / 2]; pair: ucodes = the up rows (row index + up_off) */
    const uint16_t *bs, *ubs;                      /* f16 block scales [..][in / 32] */
    long long rows_per_group; int up_off;
    int in, rows;                                  /* columns; output rows (pairs) per group, a multiple of 16 */
    int groups;                                    /* 1, or one per expert */
    int owners;                                    /* how many of them can have items, where the caller knows; 0: all, or not known */
    /* which activations: group g owns list[g * list_stride ..] of count[g] items (list NULL: items 0..M-1), or positions
     * [offset[g], offset[g + 1]) of an order sorted by group, with item = index[position] (NULL: the position) */
    const int *count, *list; int list_stride;
    const int *offset, *index, *act_index;         /* act_index: position -> activation row when it is not item / act_div */
    int M, act_div;
    const unsigned char *act;                      /* quantised rows, sp_act_pitch(in) apart: in int8 (de-interleaved by 8), then in / 16 block scales */
    /* pair: geglu(gate . x, up . x), quantised again in blocks of 16, in the same form: out_act + item * sp_act_pitch(rows);
     * otherwise out_f[item * out_stride + row] */
    unsigned char *out_act; float *out_f; int out_stride;
};

cudaError_t sp_rows_prepare();                     /* per device: the kernels' dynamic shared-memory limits */
/* one launch over `nseg` (1 or 2) segments; pair: all of them gate|up with GeGLU; items: how many the last segment's groups
 * have together */
cudaError_t sp_rows_launch(const SpRowsSeg *seg, int nseg, bool pair, long long items, int *status, cudaStream_t st, int *nl);
