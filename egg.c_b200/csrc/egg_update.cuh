// The update of a whole model in a handful of launches (egg_update.cu); declarations for the C-ABI layer.
//
// Every noise value of the update is noise(step_seed + p + seed_base + off, i) for a pair p and an index i
// (mgpu.cu:1092-1098): parameters differ only in where their window of seeds starts.  One table
//     T[i][c] = noise(step_seed + c - 16, i)
// therefore holds the noise of all of them, and a parameter's vector for pair p is column p + 16 + seed_base + off.
#pragma once

#include "egg_kernels.cuh"

#include <vector>

namespace egg {

constexpr int UPD_ORIGIN = 16;        // columns before the first seed: windows may be aligned down by up to 15

// One matrix of a batch.  The contraction index j of its vote product starts 0..15 columns before its first pair so that the
// table serves as one operand in place (a TMA copy starts on a 16-byte boundary); the other operand, fitness times noise,
// is written out with the same alignment.  Which side carries the fitness makes no difference while the products fit a byte, so
// form 0 writes the smaller of the two dimensions; where they wrap, the side is part of the result and form 1 writes the outputs n,
// as the isolated update does.
struct UpdForm {
    int fn_is_n;                      // 1: the written operand runs over the outputs n, the table over k; 0: the other way round
    int fn_row0;                      // first row of the written operand
    int x_fn;                         // table column of its contraction index 0 (any alignment)
    int x_tab, r;                     // table column of the in-place operand's index 0 (multiple of 16); index of the first pair
};
struct UpdMat {
    int rows_k, cols_n;
    UpdForm form[2];
    int tile0, tiles_n;               // first tile of the batch, tiles along k
    int blk0;                         // first block of the optimiser step
    int muon;
    float lr_scale;
    int64_t model_off, opt_off, shadow_off, votes_off, ov_in, ov_out;
};
struct UpdVec {
    int len, x_a, r;                  // x_a: table column of pair 0's first factor, aligned down by r; the second factor is one column on
    float lr_scale;
    int64_t model_off, opt_off, ov;
};
// 64 table columns that some vectors' windows cover: the first column, and which tiles of eight vectors (two words: up to 64).
struct UpdVecCols { int col; uint32_t tiles[2]; };
struct UpdHyper { float lr, beta1, beta2, eps, wd, mu; };

struct UpdBatch {
    int first, count;                 // matrices
    int tiles, splits, blocks;
    int fn_rows[2];                   // rows of the written operand in either form
    int64_t votes;                    // weights of the batch (elements of one partial vote array)
    bool any_adam;
};

// Muon-optimised matrices of one shape in one batch.
struct MuonGroup { int batch, rows, cols, first, count, slot; };      // first: position in the list; slot: workspace and side stream

// Host plan of an update over a set of parameters: batches of matrices that fit the workspace, device descriptors.
struct UpdPlan {
    int cg;                           // blocks that form a vote tile together
    std::vector<UpdMat> mats;
    std::vector<int> mat_param;       // index into the parameter list
    std::vector<UpdVec> vecs;         // the 4H-long ones first
    std::vector<UpdBatch> batches;
    std::vector<MuonGroup> groups;
    std::vector<int> list;            // matrix indices in group order
    std::vector<int2> chunks;         // table columns to fill: {first, count}, count <= UPD_CHUNK
    int W = 0, pitch = 0, kp = 0, pairs = 0;
    int vec_long = 0, len_long = 0, len_short = 0;
    int vec_pad = 0;                  // vectors rounded up to tiles of eight
    std::vector<UpdVecCols> vcols;
    int64_t fn_bytes = 0, votes_elems = 0;
    std::vector<uint8_t> descriptors; // device image of mats | vecs | chunks | list
    int64_t o_vecs = 0, o_chunks = 0, o_list = 0, o_vcols = 0;
    UpdMat *d_mats = nullptr; UpdVec *d_vecs = nullptr; int2 *d_chunks = nullptr; int *d_list = nullptr; UpdVecCols *d_vcols = nullptr;
};
constexpr int UPD_CHUNK = 1024;       // table columns per block

// use: which parameters take part (empty: all).  Host only; upd_plan_upload copies the descriptors to `dev` (as long as
// plan.descriptors), which stays the caller's.
int upd_plan_build(UpdPlan &pl, const std::vector<ParamDesc> &params, const std::vector<char> &use, int hidden, int vocab, int pairs, int num_sms);
int upd_plan_upload(UpdPlan &pl, uint8_t *dev, cudaStream_t st);
int64_t upd_table_bytes(const UpdPlan &pl);
int64_t upd_mask_bytes(const UpdPlan &pl);

int upd_init();                       // kernel attributes; once per device
// also clears what the update adds up: the change count, the wide-fitness flag and the norms of the plan's list
int launch_upd_table(cudaStream_t st, const UpdPlan &pl, int8_t *tab, uint32_t step_seed, int mask, int gaussian, unsigned long long *total, int *range,
                     double *norm2);
// masks[sign][16][kp]: bytes 0xFF where the fitness of pair (index - shift) is +1 / -1.  vfit[vec_pad][pitch]: the fitness as
// bytes, placed at every vector's own window of table columns; vvotes[vec_pad][len_long] is cleared.  *range: bit 0 when some
// |f| > 1, bit 1 when some |f| > 127, bit 2 when some |f| times the largest noise value `amp` is.
int launch_upd_masks(cudaStream_t st, const UpdPlan &pl, const int32_t *fit, uint8_t *masks, int8_t *vfit, int32_t *vvotes, int *range, int amp);
int64_t upd_vfit_bytes(const UpdPlan &pl);
int64_t upd_vvotes_elems(const UpdPlan &pl);
// votes of all vectors (noise magnitudes up to 15), then their optimiser steps
int launch_upd_vectors(cudaStream_t st, const UpdPlan &pl, const int8_t *tab, const uint8_t *masks, const int8_t *vfit, int32_t *vvotes, const int *range,
                       const int32_t *fit, int gaussian, int8_t *model, uint8_t *opt, const UpdHyper &h, unsigned long long *total, uint8_t *changed, int num_sms);
int launch_upd_operands(cudaStream_t st, const UpdPlan &pl, const UpdBatch &b, const int8_t *tab, const uint8_t *masks, const int *range,
                        const int32_t *fit, int8_t *fn);
int launch_upd_votes(cudaStream_t st, const UpdPlan &pl, const UpdBatch &b, const int8_t *tab, const int8_t *fn, const int *range, int32_t *votes, int *err, int num_sms);
int launch_upd_adam(cudaStream_t st, const UpdPlan &pl, const UpdBatch &b, const int32_t *votes, int8_t *model, uint8_t *opt, int8_t *shadow,
                    const UpdHyper &h, unsigned long long *total, uint8_t *changed);
// one pass over all overlays (update_overlay_kernel, d-eggs/src/kernels.cu:61-77); entries whose `active` byte is 0 stay as they are
int launch_overlay_step_all(cudaStream_t st, int8_t *ov, uint8_t *changed, const uint8_t *active, int n, int inc, int dec);

int upd_tensor_map(void *map, const void *ptr, uint64_t rows, uint64_t pitch, uint32_t box_rows);     // egg_gemm_inst.cu

}  // namespace egg
