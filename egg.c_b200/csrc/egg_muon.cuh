// Muon steps of batches of equally shaped matrices (egg_muon.cu).
#pragma once

#include "egg_update.cuh"

#include <cuda_bf16.h>

namespace egg {

// Workspace of a batch of nb matrices of rows x cols: the iterate as three bf16 terms in both layouts, twice (one read, one
// written), the K x K factor in three terms, and the fp32 result.
struct NsWs {
    __nv_bfloat16 *xr[2] = {nullptr, nullptr};     // [3][nb][rows][cols]
    __nv_bfloat16 *xc[2] = {nullptr, nullptr};     // [3][nb][cols][rows]
    __nv_bfloat16 *g = nullptr;                    // [3][nb][K][K], K = min(rows, cols)
    float *y = nullptr;                            // [nb][rows][cols]
    void *base = nullptr;
    int64_t bytes = 0;
};
int64_t ns_ws_bytes(int rows, int cols, int nb);
// carves the buffers out of `base` (ns_ws_bytes long)
void ns_ws_carve(NsWs &ws, void *base, int rows, int cols, int nb);

int muon_init();
// m = mu * m + vote for the listed matrices, Σ m² per matrix into norm2[list position] (cleared by the caller)
int launch_muon_momentum(cudaStream_t st, const UpdMat *mats, const int *list, int nb, int rows, int cols, const int32_t *votes, int splits,
                         int64_t split_stride, uint8_t *opt, float mu, double *norm2);
// X = m / |m| in three terms, both layouts
int launch_muon_split(cudaStream_t st, const UpdMat *mats, const int *list, int nb, int rows, int cols, const uint8_t *opt, const double *norm2, const NsWs &ws);
// five cubic Newton-Schulz steps; the result lands in ws.y
int launch_newton_schulz(cudaStream_t st, const NsWs &ws, int rows, int cols, int nb, int *err, int num_sms);
// quantised apply of ws.y; shadow may be null
int launch_muon_apply(cudaStream_t st, const UpdMat *mats, const int *list, int nb, int rows, int cols, const float *y, int8_t *model, uint8_t *opt,
                      int8_t *shadow, float lr, float wd, unsigned long long *total);

int bf16_tensor_map(void *map, const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows);     // egg_gemm_inst.cu: boxes of 64 columns x box_rows

}  // namespace egg
