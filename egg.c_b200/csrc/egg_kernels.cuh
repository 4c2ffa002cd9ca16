// Declarations shared between the kernel translation units and the C-ABI layer.
#pragma once

#include <cuda.h>
#include "egg_common.cuh"
#include "egg_gemm.cuh"

namespace egg {

// ---- per-pair noise table -------------------------------------------------
// Every noise vector a wave needs is generated once per (pair, generation) by
// the counter hash and kept in HBM/L2; the 2*seq_len rows of a pair share it.
struct NoiseSeg {
    int off;        // byte offset inside the pair's table
    int len;        // elements (a delta segment occupies 2*len bytes: [+sign][len], [-sign][len])
    int kind;       // 0: noise(S0+seed_a, i)   1: ((n(S0+seed_a,i)*n(S0+seed_b,i)*sign) >> shift) per sign, int8 [2][len]
                    // 2: model[model_off+i] + that delta, int16 [2][len] (occupies 4*len bytes)
    int seed_a, seed_b;
    int shift;
    int64_t model_off;
    int64_t scale_off;   // AdaptiveScales offset of the overlay scaling this segment (-1: raw noise)
    int first;           // index of the segment's first slice in the table-wide slice order (set by noise_index_slices)
};

// Fills NoiseSeg::first for a finished segment list and returns the total number of slices.
int noise_index_slices(NoiseSeg *segs, int nsegs);

struct NormOff { int w_m, b_m; };                       // perturbed gain / bias, int16 [2][H] each
struct MlpOff { int up_b, up_a, bup_d, dn_b, dn_a, bdn_d; };
struct LayerOff { NormOff ln1; int qkv_b; int qkv_a; int o_b, o_a; NormOff ln2; MlpOff mlp; };

struct NoiseMap {
    int64_t stride;          // bytes per pair (multiple of 16)
    int emb_a, emb_b, emb_bias_d;
    int head_a;              // emb_a scaled by the embedding_row overlay (equal to emb_a without overlays)
    NormOff ln_init, ln_f;
    MlpOff mlp_init;
    int layer0, layer_stride;   // byte offset of layer 0 block, bytes per layer block
    LayerOff layer_rel;         // offsets relative to the layer block
};

// Builds the map and the segment list for a configuration (host).
void build_noise_map(const egg_config &c, NoiseMap *map, NoiseSeg *segs, int *nsegs, int max_segs);

// Table of all distinct noise values of a wave (base null: hash every value where it is stored).
struct NoiseTable {
    int8_t *base = nullptr;
    int pitch = 0, width = 0;    // bytes per row: of the rows that also serve the embedding, of the others
    int top_seed = 0;            // largest seed offset plus one
};
int launch_noise_fill(cudaStream_t st, int8_t *nt, int64_t stride, const NoiseSeg *d_segs, int nsegs, int n_pairs,
                      uint32_t step_seed, int pair_base, int mask, int gaussian, const int8_t *model, const int8_t *scales, int32_t *loss /* cleared for every pair's two members, or null */,
                      const NoiseTable &tab = NoiseTable());

// ---- row-wise kernels -------------------------------------------------------
struct RowParams {
    int M, H, seq_len;           // seq_len: rows of one member
    int tok_len;                 // tokens of one member (<= seq_len; the rows beyond repeat the last one)
    FastDiv fd_seq;              // seq_len as a multiply-shift divisor (filled by launch_rowwise)
    const int8_t *nt; int64_t nt_stride;
    // source: embedding (mode 0), adaptive layer normalise of pre32 (mode 1), or the finished int8 stream (mode 2)
    const uint8_t *dataset; int64_t data_len, start_idx, data_stride; int pop_base, use_same_data;
    int tok_wide;                // 0: byte tokens; 1: dataset is a uint32_t array (vocab_size != 256), positions count tokens
    const int8_t *emb_rows;      // token-major copy of the embedding, [vocab][H] (the K-major shadow of the tied head)
    const int8_t *emb_bias; int vocab;
    int nt_emb_a, nt_emb_b, nt_emb_bias_d, emb_shift;
    const int8_t *ov_emb_row, *ov_emb_col;   // adaptive-noise overlays of the embedding ([vocab], [H]) or null
    const int32_t *ntt_coef;     // transformed-window coefficients [wave pairs][seq_len] (ntt_mode != 0) or null
    const int8_t *ntt_rows;      // token-major copies of ntt_emb1..3, [3][vocab][H]
    const int32_t *pre32; int32_t *rowmax;
    // residual stream out (modes 0, 1); in mode 2 the residual stream is final already and is only read, from x_out
    int8_t *x_out;
    // mean-abs norm (apply_standard_norm, mgpu.cu:646-678)
    int nt_w_m, nt_b_m;          // perturbed gain / bias tables (int16 [2][H])
    int8_t *h_out;
    // Σ_d h_d * noise_B[d] for up to three following projections
    int ndots; int nt_dot[3]; int32_t *xb_out; int xb_stride;
    // accumulators to clear for the kernels that follow
    int32_t *zero1;      // [M]
    int32_t *zero2;      // [M]
    int32_t *zero3;      // [M][3]
    int one;             // 1 (filled by launch_rowwise): the multiplier of additions issued as multiply-adds
};
int launch_rowwise(cudaStream_t st, const RowParams &p, int mode);

// Σ x·noise·factor per row under adaptive-noise overlays; overwrites out[r*out_stride + q].
struct ScaledDotParams {
    int M, H, seq_len;
    FastDiv fd_seq;              // filled by launch_scaled_dot
    int terms;                   // 1: x is [M][H];  4: x is [M][4H], four terms per thread summed with a running truncation
    const int8_t *x;
    const int8_t *nt; int64_t nt_stride;
    int ndots; int nt_dot[3];    // offsets of the raw noise vectors (length H*terms) in the pair table
    const int8_t *ov[3];         // overlays over the input index (length H*terms)
    int32_t *out; int out_stride;
};
int launch_scaled_dot(cudaStream_t st, const ScaledDotParams &p);

struct AqnParams {
    int M, H;
    const int32_t *pre3;      // [M][3H]
    const int32_t *rowmax3;   // [M][3]
    int8_t *q, *k, *v;        // [M][H] each
};
int launch_aqn(cudaStream_t st, const AqnParams &p);

struct AttnParams {
    int members, H, head_dim, seq_len, shift_attn;
    int row_stride;           // rows of one member in the buffers below (>= seq_len)
    const int8_t *q, *k, *v;  // [members*row_stride][H]
    int8_t *ao;               // [members*row_stride][H]
    const int32_t *exp_lut;
    const int8_t *nt; int64_t nt_stride; int nt_o_b;
    int32_t *xbo;             // [members*seq_len] += Σ_d ao_d * noise_B_o[d]
};
int launch_attention(cudaStream_t st, const AttnParams &p);
// scores, weights and sums in tensor memory (egg_attention_tm.cu)
bool attention_tm_supported(int seq_len, int row_stride);
int launch_attention_tm(cudaStream_t st, const AttnParams &p, int num_sms, int *err);
// the same attention on tcgen05 (egg_attention_tc.cu): whole 128-query blocks of one member, head_dim 64, seq_len <= 512
bool attention_tc_supported(int seq_len, int head_dim);
int launch_attention_tc(cudaStream_t st, const AttnParams &p, int *err);
// scores on mma.sync per warp, Σ wt·v on tcgen05 with the accumulators in tensor memory (egg_attention_tc.cu)
int launch_attention_hy(cudaStream_t st, const AttnParams &p, int *err);

// ---- sampling -----------------------------------------------------------------
struct GenParams {
    int H, V, head_dim, n_layers;
    int shift_attn, shift_out, shift_logit, shift_mlp_up, shift_mlp_down, rope_bit;
    const int8_t *model; ModelLayout L;
    const int8_t *act_lut; const int32_t *exp_lut; const int32_t *rope_lut;
    // K-major weight copies, [N][K]; per layer at w_layer0 + l * w_layer_stride: q|k|v, output, MLP up, MLP down
    const int8_t *w_init_up, *w_init_dn, *w_emb, *w_layer0; int64_t w_layer_stride, w_qkv, w_o, w_up, w_dn;
    int8_t *kv;                  // [n_layers][heads][2][256][64]
    int *err;
    uint8_t *tokens;             // [256]: first seed_len given, up to seed_len + gen_len written
    int seed_len, gen_len;
    int start;                   // first token to process: the cache holds the ones before
    uint32_t seed;
    float temp; int filter, min_p_limit, penalty_int;
    int scan_block;              // block size of the reference kernel: fixes the order of its weighted draw
};
int launch_generate(cudaStream_t st, const GenParams &p);
// one layer's cache [heads][2][256][64] from the first `count` rows of k and v, [rows][H]
int launch_kv_gather(cudaStream_t st, const int8_t *k, const int8_t *v, int H, int count, int8_t *kv);

// ---- weights ----------------------------------------------------------------
// packed [K/4][N][4] -> K-major shadow [N][K]
int launch_unpack_transpose(cudaStream_t st, const int8_t *packed, int8_t *shadow, int rows_k, int cols_n);

// ---- row-owning GEMM with the adaptive normalisation fused (egg_gemm_fused.cuh) -----
struct FusedParams;
// mode: FUSED_QKV (out = [3][part_rows][H] int8: q, k, v) or FUSED_RES (out = x [M][H] int8, resid = x, may alias out)
int launch_gemm_fused(cudaStream_t st, int mode, const int8_t *A, const int8_t *B, int8_t *out, const int8_t *resid,
                      const FusedParams &p, int num_sms);
// whether the row-owning kernels can run a configuration (whole 32-row groups of one member, a row fits tensor memory)
int fused_cluster_size(int hidden);       // blocks per unit of the row-owning GEMM (two also where units are few), 0 when the width is unsupported
inline bool fused_supported(int hidden, int seq_len) { return seq_len % 32 == 0 && fused_cluster_size(hidden) > 0; }
// Largest output shift + rank-1 shift of the projections that add their bias before both (the row-owning residual projections
// and MLP-up): (bias + noise) << (both shifts) joins a product below 2^30.
constexpr int PRESHIFT_MAX = 20;
// 2^rank1_shift where the rank-1 shift t and the output shift s of a projection over K may be merged into one, else 0:
// |acc| * 2^t + |xb * a| + |(bias + noise) << (s + t)| < 2^31 for every input.  |acc| <= K * 127 * 128 (activations are clipped to
// 127, a weight may be -128), |xb| <= K * 127 * 45, |a| <= 45 (three noise values of mask 15 added), |bias + noise| <= 256.
inline int merged_shift(int K, int rank1_shift, int out_shift) {
    if (rank1_shift > PRESHIFT_MAX || out_shift > PRESHIFT_MAX) return 0;
    const int64_t bound = (int64_t)K * 127 * 128 * (1ll << rank1_shift) + (int64_t)K * 127 * 45 * 45 + (256ll << (out_shift + rank1_shift));
    return bound < (1ll << 31) ? 1 << rank1_shift : 0;
}
// Rows that hold one member's seq_len tokens: padded to whole 32-row groups where that opens the row-owning kernels and the
// row-per-lane epilogues for at most a third more rows (48 -> 64 costs 1.33; 16 -> 32 would double the work).
inline int member_rows(int hidden, int seq_len) {
    const int up = (seq_len + 31) / 32 * 32;
    return fused_cluster_size(hidden) > 0 && 3 * up <= 4 * seq_len ? up : seq_len;
}

// ---- GEMM -------------------------------------------------------------------
// A: [M][K] int8 row-major, B: [N][K] int8 row-major (both device pointers).
int launch_gemm(cudaStream_t st, int epi, const int8_t *A, const int8_t *B, const GemmParams &p, int num_sms);
int gemm_init();   // resolves the driver entry point for tensor-map encoding, sets smem attributes

// ---- fitness / update -------------------------------------------------------
// Transform of every pair's input window (ntt_mode 1..3): see window_transform_kernel.
struct WindowParams {
    int mode, seq_len, pairs;
    const uint8_t *dataset; int tok_wide; int64_t data_len, start_idx, data_stride; int pair_base, use_same_data;
    int32_t *coef;               // [pairs][seq_len]
};
int launch_window_transform(cudaStream_t st, const WindowParams &p);
// Second pass of the head over the bytes and maxima that EPI_LOGITS leaves (vocab_size != 256): see head_loss_kernel.
struct HeadLossParams {
    int M, V, H, seq_len, tok_len;  // rows and tokens of one member
    FastDiv fd_seq;              // filled by launch_head_loss
    const uint8_t *below;        // [M][V] min(255, maximum of the 64 - logit), logits after >> SHIFT_LOGIT
    const int32_t *max64;        // [M][V/64] those maxima
    // what the target's logit is computed from
    const int8_t *h, *emb; const int32_t *xb; int xb_stride; const int8_t *nt; int64_t nt_stride; int nt_a_off, rank1_shift, out_shift;
    const int32_t *exp_lut;      // 256
    const uint32_t *dataset; int64_t data_len, start_idx, data_stride; int pop_base, use_same_data;
    int softmax_scale_bit;
    int32_t *loss;               // [wave members] +=
};
int launch_head_loss(cudaStream_t st, const HeadLossParams &p, int num_sms);
int launch_fitness(cudaStream_t st, const int32_t *loss, int32_t *fit, int pairs, int32_t *copy = nullptr /* pinned host memory for the losses */);
int launch_publish(cudaStream_t st, void *dst /* pinned host memory */, const void *src);      // 16 bytes

// operand generation for the update GEMM: NA[n][Kp] = f_p * noise(s_p+off_a, n), NB[k][Kp] = noise(s_p+off_b, k)
// split = 1 doubles the contraction: [f0*a | f1*a] x [b ; 16 b] with f = 16 f1 + f0.
int launch_update_operands(cudaStream_t st, int8_t *na, int8_t *nb, const int32_t *fit, int pairs, int kp, int rows_k,
                           int cols_n, int off_a, int off_b, int seed_base, uint32_t step_seed, int mask, int gaussian,
                           int split);

// Splits of the pair index for the vote GEMM of a rows_k x cols_n matrix over kp (padded) pairs: enough work items to
// fill the GPU twice over, never an empty split.
int vote_gemm_splits(int rows_k, int cols_n, int kp, int num_sms);

// Optimiser step of one matrix from its (partial) vote matrices, element order = the packed weight layout.
struct VoteApplyParams {
    int8_t *w_packed;            // [rows_k/4][cols_n][4]
    float *opt;                  // AdamParam{m,v,acc} per packed index
    const int32_t *votes;        // [nsplits][rows_k * cols_n]
    int nsplits; int64_t split_stride;
    int rows_k, cols_n;
    float lr, beta1, beta2, eps, wd;
    unsigned long long *total_updates;
};
int launch_adam_from_votes(cudaStream_t st, const VoteApplyParams &p);        // ES-AdamW (mgpu.cu:1040-1064, 1100-1110)

}  // namespace egg
