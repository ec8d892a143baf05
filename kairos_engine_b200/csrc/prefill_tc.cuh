/* prefill_tc.cuh — launch interface of the tensor-core prefill GEMMs (prefill_tc.cu): grouped
 * Q4B-weight x fp16-split-activation GEMMs on tcgen05 with TMEM accumulators. */
#pragma once
#include "common.cuh"

struct SpTcPlan;     /* buffers, tile tables and TMA descriptors; host object */

/* K dimensions must be multiples of 64 (one 128-byte swizzled shared-memory row of fp16) */
bool sp_tc_supported(const SpDims &d);
cudaError_t sp_tc_create(const SpDims &d, int max_tokens, int max_rows, SpTcPlan **out, size_t *bytes);
void sp_tc_destroy(SpTcPlan *p);

/* shared expert: nx [M][E] f32 (normalised input) -> dn [M][E] f32 = Wd . geglu(Wg nx, Wu nx) */
cudaError_t sp_tc_shared_expert(SpTcPlan *p, const SpDims &d, const SpLayerDev &L, int M, const float *nx, float *dn,
                                int *status, cudaStream_t st, int *nl, int phase = 0);
/* routed experts on R rows sorted by expert (expert e owns rows [offsets[e], offsets[e+1]), device
 * array of NE+1 ints): out[rowmap ? rowmap[r] : r][E] = Wdn[e] . geglu(Wgu[e] . rows[r]).
 * gather != NULL: row r is src[gather[r]] instead of src[r]. R <= max_rows. owners: how many experts the rows can belong to, 0 =
 * not known. */
cudaError_t sp_tc_routed(SpTcPlan *p, const SpDims &d, const SpLayerDev &L, int R, int owners, const float *src, const int *gather,
                         const int *offsets, const int *rowmap, float *out, int *status, cudaStream_t st, int *nl);
/* one whole layer's GEMMs on one GPU, the shared expert and the routed experts in one launch each for gate|up and down:
 * sel_asc / pairpos [M*NU] and count [NE] from the selection -> dn [M][E], eo [M*NU][E] (row = pair). The experts' normalised
 * inputs [M][E] are written beforehand into sp_tc_inputs' rows as fp16 hi/lo (k order 0,4,1,5,2,6,3,7 in each group of 8). */
void sp_tc_inputs(SpTcPlan *p, __half **nx_hi, __half **nx_lo, __half **in_hi, __half **in_lo);
cudaError_t sp_tc_layer(SpTcPlan *p, const SpDims &d, const SpLayerDev &L, int M, const int *sel_asc, const int *count, const int *pairpos, float *dn, float *eo,
                        int *status, cudaStream_t st, int *nl);
