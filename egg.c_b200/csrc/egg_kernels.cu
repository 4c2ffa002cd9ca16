// Non-GEMM kernels of the evaluation: per-pair noise tables, row-wise embedding /
// adaptive-normalise / mean-abs-norm, Q/K/V requantisation, causal integer-softmax
// attention, cross-entropy, fitness; operands and AdamW of the isolated update.  "mgpu.cu" = full_cuda_train_transformer_adam_mgpu.cu.
#include "egg_kernels.cuh"

#include <limits.h>

namespace egg {

// =========================================================================
// noise table
// =========================================================================

void build_noise_map(const egg_config &c, NoiseMap *map, NoiseSeg *segs, int *nsegs, int max_segs) {
    const int H = c.hidden_dim, V = c.vocab_size;
    const int ssv = c.sigma_shift_vector;
    const ScalesLayout SL = scales_layout(c);
    int n = 0, off = 0;
    // sc = AdaptiveScales offset of the overlay that scales the segment (-1: the segment holds raw noise)
    auto put = [&](int kind, int len, int sa, int sb, int shift, int64_t moff, int64_t sc, int bytes) {
        int o = off;
        if (n < max_segs) { segs[n] = NoiseSeg{off, len, kind, sa, sb, shift, moff, sc}; }
        n++; off += bytes; return o;
    };
    auto plain = [&](int len, int seed, int64_t sc) { return put(0, len, seed, 0, 0, -1, sc, len); };
    auto delta = [&](int len, int sa, int sb, int64_t sc) { return put(1, len, sa, sb, ssv, -1, sc, 2 * len); };
    // kind 2: model byte + delta, both signs, as int16 [2][len] (4*len bytes); moff = element offset in TransformerModel
    auto comb = [&](int len, int sa, int sb, int64_t moff, int64_t sc) { return put(2, len, sa, sb, ssv, moff, sc, 4 * len); };
    auto norm = [&](int base, int wa, int wb, int ba, int bb, int64_t mw, int64_t mb, int64_t sw, int64_t sbias) {
        NormOff r; r.w_m = comb(H, base + wa, base + wb, mw, sw); r.b_m = comb(H, base + ba, base + bb, mb, sbias); return r;
    };
    auto mlp = [&](int base, int up_a, int up_b, int bu_a, int bu_b, int dn_a, int dn_b, int bd_a, int bd_b, int64_t s_up_col,
                   int64_t s_bup, int64_t s_dn_col, int64_t s_bdn) {
        MlpOff r;
        r.up_b = plain(H, base + up_b, -1);
        r.up_a = plain(4 * H, base + up_a, s_up_col);
        r.bup_d = delta(4 * H, base + bu_a, base + bu_b, s_bup);
        r.dn_b = plain(4 * H, base + dn_b, -1);
        r.dn_a = plain(H, base + dn_a, s_dn_col);
        r.bdn_d = delta(H, base + bd_a, base + bd_b, s_bdn);
        return r;
    };
    // seed offsets: mgpu.cu:114-165.  Vectors that feed a row dot (the "B" side) stay raw: their overlay is
    // applied per term of the dot.  emb_a is read raw by the embedding and scaled (head_a) by the head.
    map->emb_a = plain(V, 0, -1);
    map->head_a = plain(V, 0, SL.embedding_row);
    map->emb_b = plain(H, 0 + H, -1);
    map->emb_bias_d = delta(H, 50, 51, SL.emb_bias);
    const ModelLayout ML = model_layout(c);
    map->ln_init = norm(0, 500, 501, 502, 503, ML.ln_init, ML.ln_init_bias, SL.ln_init, SL.ln_init_bias);
    map->ln_f = norm(0, 900, 901, 910, 911, ML.ln_f, ML.ln_f_bias, SL.ln_f, SL.ln_f_bias);
    map->mlp_init = mlp(0, 510, 511, 514, 515, 512, 513, 516, 517, SL.w_emb_mlp_up_col, SL.mlp_emb_bias_up, SL.w_emb_mlp_down_col,
                        SL.mlp_emb_bias_down);
    map->layer0 = off;
    for (int l = 0; l < c.n_layers; l++) {
        int base = l * 1000, start = off;
        const int64_t lH = (int64_t)l * H;
        LayerOff lo;
        lo.ln1 = norm(base, 100, 101, 110, 111, ML.ln_1 + lH, ML.ln_1_bias + lH, SL.ln_1 + lH, SL.ln_1_bias + lH);
        lo.qkv_b = plain(H, base + 201, -1); plain(H, base + 203, -1); plain(H, base + 205, -1);
        lo.qkv_a = plain(H, base + 200, SL.w_q_col + lH); plain(H, base + 202, SL.w_k_col + lH); plain(H, base + 204, SL.w_v_col + lH);
        lo.o_b = plain(H, base + 207, -1);
        lo.o_a = plain(H, base + 206, SL.w_o_col + lH);
        lo.ln2 = norm(base, 300, 301, 310, 311, ML.ln_2 + lH, ML.ln_2_bias + lH, SL.ln_2 + lH, SL.ln_2_bias + lH);
        lo.mlp = mlp(base, 400, 401, 410, 411, 402, 403, 412, 413, SL.w_up_col + 4 * lH, SL.mlp_bias_up + 4 * lH, SL.w_down_col + lH,
                     SL.mlp_bias_down + lH);
        if (l == 0) {
            map->layer_stride = off - start;
            LayerOff rel = lo;
            int *pi = reinterpret_cast<int *>(&rel);
            for (size_t i = 0; i < sizeof(LayerOff) / sizeof(int); i++) pi[i] -= start;
            map->layer_rel = rel;
        }
    }
    map->stride = (off + 15) & ~15;
    *nsegs = n;
    noise_index_slices(segs, n < max_segs ? n : max_segs);
}

__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d);

// scales: AdaptiveScales bytes or null.  With scales, every segment that has an overlay holds
// (int)(noise * factor) (A vectors, layers.cuh:90) or the delta built from (int)(n1 * n2 * factor)
// (vectors, layers.cuh:176-180), so that the consumers of the table need not know about overlays.
constexpr int NOISE_SLICE = 128;       // elements per warp and step: every segment length is a multiple of it

int noise_index_slices(NoiseSeg *segs, int nsegs) {
    int acc = 0;
    for (int i = 0; i < nsegs; i++) { segs[i].first = acc; acc += (segs[i].len + NOISE_SLICE - 1) / NOISE_SLICE; }
    return acc;
}

// The pairs of a wave and the vectors of a pair only shift the seed: noise(S0 + pair + seed, i).  For many pairs each distinct
// (seed, index) is hashed once into tab[pair + seed][i] and the pairs' tables are filled from there: 4096 pairs at H 256, 4 layers
// take 8 million hashes instead of 280.  Rows below `wide_rows` hold the embedding's noise and are `pitch` long, the others 4 H.
__global__ void __launch_bounds__(256) noise_table_kernel(int8_t *tab, int pitch, int width, int rows, int wide_rows, uint32_t seed0, int mask, int gaussian) {
    chain_next();
    chain_wait();
    const int row = blockIdx.x;
    const int n = row < wide_rows ? pitch : width;
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) {
        int v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = noise_from_hash(seed0 + (uint32_t)row, (uint32_t)(i + e), mask, gaussian);
        *reinterpret_cast<uint32_t *>(tab + (int64_t)row * pitch + i) = pack4(v[0], v[1], v[2], v[3]);
    }
}

// One element of a segment for both signs of a pair: an A vector's noise, or the delta of a product of two (plus the parameter).
__device__ __forceinline__ void noise_element(const NoiseSeg &sg, int i, int val, const int8_t *scales, int &vp, int &vn) {
    if (scales) val = scale_trunc(val, overlay_num(scales[sg.scale_off + i]));
    vp = sg.kind == 0 ? val : val >> sg.shift;
    vn = (-val) >> sg.shift;
}

__global__ void __launch_bounds__(256) noise_fill_kernel(int8_t *nt, int64_t stride, const NoiseSeg *segs, int nsegs, uint32_t step_seed,
                                                         int pair_base, int mask, int gaussian, const int8_t *model, const int8_t *scales, int32_t *loss) {
    chain_next();
    chain_wait();
    if (loss && blockIdx.x == 0 && threadIdx.x < 2) loss[2 * blockIdx.y + threadIdx.x] = 0;      // the pair's losses start here
    extern __shared__ NoiseSeg s_segs[];
    for (int i = threadIdx.x; i < nsegs; i += blockDim.x) s_segs[i] = segs[i];
    __syncthreads();
    const int total_slices = s_segs[nsegs - 1].first + (s_segs[nsegs - 1].len + NOISE_SLICE - 1) / NOISE_SLICE;
    const int pair = blockIdx.y;
    const uint32_t S0 = step_seed + (uint32_t)(pair_base + pair);
    int8_t *dst = nt + (int64_t)pair * stride;
    // one warp step = 128 consecutive elements of one segment, four per lane; an element of a delta segment is hashed once and
    // written for both signs.  Consecutive warps take consecutive slices.
    int g = 0;
    for (int sl = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)); sl < total_slices; sl += (int)(gridDim.x * (blockDim.x >> 5))) {
        while (g + 1 < nsegs && s_segs[g + 1].first <= sl) g++;    // slices are visited in increasing order
        const NoiseSeg sg = s_segs[g];
        const int i0 = (sl - sg.first) * NOISE_SLICE + ((threadIdx.x & 31) << 2);
        if (i0 >= sg.len) continue;
        const int8_t *ov = sg.scale_off >= 0 ? scales : nullptr;
        int vp[4], vn[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int i = i0 + e;
            int val = noise_from_hash(S0 + (uint32_t)sg.seed_a, (uint32_t)i, mask, gaussian);
            if (sg.kind != 0) val *= noise_from_hash(S0 + (uint32_t)sg.seed_b, (uint32_t)i, mask, gaussian);
            noise_element(sg, i, val, ov, vp[e], vn[e]);
            if (sg.kind == 2) { const int m = model[sg.model_off + i]; vp[e] += m; vn[e] += m; }
        }
        if (sg.kind == 2) {
            int16_t *d16 = reinterpret_cast<int16_t *>(dst + sg.off);
            *reinterpret_cast<int2 *>(d16 + i0) = make_int2((vp[0] & 0xFFFF) | (vp[1] << 16), (vp[2] & 0xFFFF) | (vp[3] << 16));
            *reinterpret_cast<int2 *>(d16 + sg.len + i0) = make_int2((vn[0] & 0xFFFF) | (vn[1] << 16), (vn[2] & 0xFFFF) | (vn[3] << 16));
        } else {
            *reinterpret_cast<uint32_t *>(dst + sg.off + i0) = pack4(vp[0], vp[1], vp[2], vp[3]);
            if (sg.kind == 1) *reinterpret_cast<uint32_t *>(dst + sg.off + sg.len + i0) = pack4(vn[0], vn[1], vn[2], vn[3]);
        }
    }
}

// The same from the wave's table, 16 elements per lane: eight lanes take a slice, a warp four (segments, offsets and the model's
// vectors start at multiples of 128 elements).  It waits for loads from L2, so wide ones
// count: a wave of 4096 pairs at H 256, 4 layers took 260 us hashed pair by pair, 160 with 4 elements per lane and 128 so, table included.
__global__ void __launch_bounds__(256) noise_fill_tab_kernel(int8_t *nt, int64_t stride, const NoiseSeg *segs, int nsegs, const int8_t *tab, int pitch, const int8_t *model,
                                                             const int8_t *scales, int32_t *loss) {
    chain_next();
    chain_wait();
    if (loss && blockIdx.x == 0 && threadIdx.x < 2) loss[2 * blockIdx.y + threadIdx.x] = 0;
    extern __shared__ NoiseSeg s_segs[];
    for (int i = threadIdx.x; i < nsegs; i += blockDim.x) s_segs[i] = segs[i];
    __syncthreads();
    const int total_slices = s_segs[nsegs - 1].first + (s_segs[nsegs - 1].len + NOISE_SLICE - 1) / NOISE_SLICE;
    const int pair = blockIdx.y;
    int8_t *dst = nt + (int64_t)pair * stride;
    int g = 0;
    for (int sl = (int)(blockIdx.x * (blockDim.x >> 3) + (threadIdx.x >> 3)); sl < total_slices; sl += (int)(gridDim.x * (blockDim.x >> 3))) {
        while (g + 1 < nsegs && s_segs[g + 1].first <= sl) g++;
        const NoiseSeg sg = s_segs[g];
        const int i0 = (sl - sg.first) * NOISE_SLICE + ((threadIdx.x & 7) << 4);
        if (i0 >= sg.len) continue;
        const int8_t *ov = sg.scale_off >= 0 ? scales : nullptr;
        const int4 a = *reinterpret_cast<const int4 *>(tab + (int64_t)(pair + sg.seed_a) * pitch + i0);
        if (sg.kind == 0 && !ov) { *reinterpret_cast<int4 *>(dst + sg.off + i0) = a; continue; }
        int4 b = make_int4(0, 0, 0, 0), m = b;
        if (sg.kind != 0) b = *reinterpret_cast<const int4 *>(tab + (int64_t)(pair + sg.seed_b) * pitch + i0);
        if (sg.kind == 2) m = *reinterpret_cast<const int4 *>(model + sg.model_off + i0);
        const int32_t wa[4] = {a.x, a.y, a.z, a.w}, wb[4] = {b.x, b.y, b.z, b.w}, wm[4] = {m.x, m.y, m.z, m.w};
        uint32_t p8[4], n8[4], p16[8], n16[8];
#pragma unroll
        for (int w = 0; w < 4; w++) {
            int vp[4], vn[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                int val = (int8_t)(wa[w] >> (8 * e));
                if (sg.kind != 0) val *= (int8_t)(wb[w] >> (8 * e));
                noise_element(sg, i0 + 4 * w + e, val, ov, vp[e], vn[e]);
                vp[e] += (int8_t)(wm[w] >> (8 * e)); vn[e] += (int8_t)(wm[w] >> (8 * e));
            }
            if (sg.kind == 2) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    p16[2 * w + e] = __byte_perm(vp[2 * e], vp[2 * e + 1], 0x5410);
                    n16[2 * w + e] = __byte_perm(vn[2 * e], vn[2 * e + 1], 0x5410);
                }
            } else {
                p8[w] = pack4(vp[0], vp[1], vp[2], vp[3]); n8[w] = pack4(vn[0], vn[1], vn[2], vn[3]);
            }
        }
        if (sg.kind == 2) {
            int16_t *d16 = reinterpret_cast<int16_t *>(dst + sg.off) + i0;
#pragma unroll
            for (int w = 0; w < 2; w++) {
                reinterpret_cast<uint4 *>(d16)[w] = make_uint4(p16[4 * w], p16[4 * w + 1], p16[4 * w + 2], p16[4 * w + 3]);
                reinterpret_cast<uint4 *>(d16 + sg.len)[w] = make_uint4(n16[4 * w], n16[4 * w + 1], n16[4 * w + 2], n16[4 * w + 3]);
            }
        } else {
            *reinterpret_cast<uint4 *>(dst + sg.off + i0) = make_uint4(p8[0], p8[1], p8[2], p8[3]);
            if (sg.kind == 1) *reinterpret_cast<uint4 *>(dst + sg.off + sg.len + i0) = make_uint4(n8[0], n8[1], n8[2], n8[3]);
        }
    }
}

int launch_noise_fill(cudaStream_t st, int8_t *nt, int64_t stride, const NoiseSeg *d_segs, int nsegs, int n_pairs,
                      uint32_t step_seed, int pair_base, int mask, int gaussian, const int8_t *model, const int8_t *scales, int32_t *loss, const NoiseTable &tab) {
    // a few slices per warp amortise the segment-table load; few pairs spread over more blocks
    int gx = (int)((stride / NOISE_SLICE + 31) / 32);
    while (gx > 1 && (int64_t)gx * n_pairs > 4096) gx >>= 1;
    if ((int64_t)gx * n_pairs < 512) gx *= 4;
    dim3 grid((unsigned)gx, (unsigned)n_pairs);
    const size_t smem = nsegs * sizeof(NoiseSeg);
    if (tab.base) {
        const int rows = n_pairs + tab.top_seed;
        EGG_CUDA(launch_chained(noise_table_kernel, rows, tab.width / 4 < 256 ? tab.width / 4 : 256, 0, st, tab.base, tab.pitch, tab.width, rows, n_pairs,
                                step_seed + (uint32_t)pair_base, mask, gaussian));
        EGG_CUDA(launch_chained(noise_fill_tab_kernel, grid, 256, smem, st, nt, stride, d_segs, nsegs, tab.base, tab.pitch, model, scales, loss));
        return EGG_OK;
    }
    EGG_CUDA(launch_chained(noise_fill_kernel, grid, 256, smem, st, nt, stride, d_segs, nsegs, step_seed, pair_base, mask, gaussian, model, scales, loss));
    return EGG_OK;
}

// =========================================================================
// row-wise: embedding | adaptive layer normalise -> x ; mean-abs norm -> h ; noise dots
// =========================================================================

__device__ __forceinline__ int warp_sum(int v) {
    return __reduce_add_sync(0xFFFFFFFFu, v);       // one warp-wide integer reduction instruction; every lane gets the sum
}

__device__ __forceinline__ int8_t byte_of(int32_t w, int i) { return (int8_t)(w >> (8 * i)); }
__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
    return (uint32_t)(a & 0xFF) | ((uint32_t)(b & 0xFF) << 8) | ((uint32_t)(c & 0xFF) << 16) | ((uint32_t)(d & 0xFF) << 24);
}

// One warp per run of ROW_RUN consecutive rows of ONE population member (seq_len is a multiple of 16, so a run never
// crosses members); NJ = H/128 chunks of 4 elements per lane.  Everything that depends on the member only -- the
// perturbed gain / bias tables and the noise vectors of the following projections, 3.5 H bytes -- is loaded once per
// run and kept in registers; per row only the row itself is read, and the next row's bytes are requested before the
// current row is worked on (mode 2), so that the warp always has a load in flight.
constexpr int ROW_RUN = 8;
#ifndef ROW_EMB_BLOCKS
#define ROW_EMB_BLOCKS 2          // resident blocks asked for in embedding mode (its per-member tables are the widest)
#endif

// WIDE (embedding mode only): the dataset holds uint32_t tokens below 65536 (vocab_size != 256, mgpu.cu:58-66)
// NTT (embedding mode only): bytes 1..3 of the row's transformed-window coefficient index three more tables whose
// rows are added >> 2 each (NTT_MODE != 0, mgpu.cu:916-929)
template <int MODE, int NJ, int NDOTS, bool WIDE = false, bool NTT = false>
__global__ void __launch_bounds__(256, MODE == 0 ? ROW_EMB_BLOCKS : 1) rowwise_kernel(const RowParams p) {
    chain_next();
    chain_wait();
    const int run = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int r0 = run * ROW_RUN;
    if (r0 >= p.M) return;
    const int r_end = min(r0 + ROW_RUN, p.M);
    const int H = NJ * 128;
    const int mem = fast_div(r0, p.fd_seq);
    const int sgn = mem & 1, ns = sgn ? -1 : 1;
    const int8_t *ntp = p.nt + (int64_t)(mem >> 1) * p.nt_stride;
    const int16_t *wm = reinterpret_cast<const int16_t *>(ntp + p.nt_w_m) + sgn * H;   // w + ((n1*n2*sign)>>SSV)
    const int16_t *bm = reinterpret_cast<const int16_t *>(ntp + p.nt_b_m) + sgn * H;

    // ---- per-member tables: gains and biases widened once per run, not once per row ----
    int wv[NJ][4], bv[NJ][4];
    int32_t n4[NDOTS][NJ];
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int d = (j << 7) + (lane << 2);
        const int2 w4 = *reinterpret_cast<const int2 *>(wm + d);
        const int2 b4 = *reinterpret_cast<const int2 *>(bm + d);
        // low halves sign-extended by one byte permute (selector msb = replicate the byte's sign), high halves by a shift
        wv[j][0] = ptx::sx_half0(w4.x); wv[j][1] = w4.x >> 16; wv[j][2] = ptx::sx_half0(w4.y); wv[j][3] = w4.y >> 16;
        bv[j][0] = ptx::sx_half0(b4.x); bv[j][1] = b4.x >> 16; bv[j][2] = ptx::sx_half0(b4.y); bv[j][3] = b4.y >> 16;
#pragma unroll
        for (int q = 0; q < NDOTS; q++) n4[q][j] = *reinterpret_cast<const int32_t *>(ntp + p.nt_dot[q] + d);
    }
    // embedding mode: bias + bias-noise delta, the B-noise of the embedding's rank-1 term and the column overlays of the run's member
    int emb_add[MODE == 0 ? NJ : 1][4];
    int32_t emb_nb[MODE == 0 ? NJ : 1], emb_oc[MODE == 0 ? NJ : 1];
    if (MODE == 0) {
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int d = (j << 7) + (lane << 2);
            const int32_t eb4 = *reinterpret_cast<const int32_t *>(p.emb_bias + d);
            const int32_t dl4 = *reinterpret_cast<const int32_t *>(ntp + p.nt_emb_bias_d + sgn * H + d);
#pragma unroll
            for (int i = 0; i < 4; i++) emb_add[j][i] = (int)byte_of(eb4, i) + (int)byte_of(dl4, i);
            emb_nb[j] = *reinterpret_cast<const int32_t *>(ntp + p.nt_emb_b + d);
            emb_oc[j] = p.ov_emb_col ? *reinterpret_cast<const int32_t *>(p.ov_emb_col + d) : 0;
        }
    }
    uint32_t xw_next[NJ];
    if (MODE == 2) {
#pragma unroll
        for (int j = 0; j < NJ; j++) xw_next[j] = *reinterpret_cast<const uint32_t *>(p.x_out + (int64_t)r0 * H + (j << 7) + (lane << 2));
    }

    // embedding mode: the run's tokens and their A-noise bytes are fetched up front (two dependent loads that would
    // otherwise sit at the head of every row), and the embedding row of the next token is requested a row ahead
    unsigned long long toks = 0, atoks = 0;          // one byte per row of the run (ROW_RUN = 8)
    unsigned long long toks_hi = 0;                  // WIDE: bits 8..15 of the run's tokens, packed the same way
    auto tok_of = [&](int i) { return (int)((toks >> (8 * i)) & 0xFF) | (WIDE ? (int)((toks_hi >> (8 * i)) & 0xFF) << 8 : 0); };
    int32_t e4_next[MODE == 0 ? NJ : 1];
    if (MODE == 0) {
        static_assert(ROW_RUN == 8, "the run's tokens are packed into one 64-bit register");
        const int64_t pair = (p.pop_base + mem) >> 1;
        const int64_t pos = p.use_same_data ? (p.start_idx % (p.data_len - p.tok_len))
                                            : ((p.start_idx + pair * p.data_stride) % (p.data_len - p.tok_len));
        const int t0 = r0 - mem * p.seq_len;
#pragma unroll
        for (int i = 0; i < ROW_RUN; i++) {
            unsigned tok = 0u;
            const int64_t at = pos + min(t0 + i, p.tok_len - 1);
            if (r0 + i < r_end) tok = WIDE ? reinterpret_cast<const uint32_t *>(p.dataset)[at] : (unsigned)p.dataset[at];
            toks |= (unsigned long long)(tok & 0xFF) << (8 * i);
            if (WIDE) toks_hi |= (unsigned long long)((tok >> 8) & 0xFF) << (8 * i);
        }
#pragma unroll
        for (int i = 0; i < ROW_RUN; i++) atoks |= (unsigned long long)(uint8_t)ntp[p.nt_emb_a + tok_of(i)] << (8 * i);
#pragma unroll
        for (int j = 0; j < NJ; j++) e4_next[j] = *reinterpret_cast<const int32_t *>(p.emb_rows + (int64_t)tok_of(0) * H + (j << 7) + (lane << 2));
    }

    for (int ri = 0; ri < ROW_RUN; ri++) {
        const int r = r0 + ri;
        if (r >= r_end) break;
        int x[NJ][4];
        uint32_t xw_cur[MODE == 2 ? NJ : 1];
        if (MODE == 0) {
            // embedding (mgpu.cu:902-931): the token's row comes from the token-major copy of the table ([V][H], the same
            // K-major shadow the head projection multiplies with), 4 contiguous bytes per lane and chunk
            const int tok = tok_of(ri);
            const int a_tok = (int)(int8_t)((atoks >> (8 * ri)) & 0xFF);
            const float f_row = p.ov_emb_row ? __fdiv_rn((float)overlay_num(p.ov_emb_row[tok]), 64.0f) : 1.0f;
            int32_t e4c[NJ];
#pragma unroll
            for (int j = 0; j < NJ; j++) e4c[j] = e4_next[j];
            if (ri + 1 < ROW_RUN && r + 1 < r_end) {
#pragma unroll
                for (int j = 0; j < NJ; j++) e4_next[j] = *reinterpret_cast<const int32_t *>(p.emb_rows + (int64_t)tok_of(ri + 1) * H + (j << 7) + (lane << 2));
            }
            int ex[NTT ? NJ : 1][4];
            if (NTT) {
                const int cw = p.ntt_coef[(int64_t)(mem >> 1) * p.seq_len + (r - mem * p.seq_len)];
#pragma unroll
                for (int j = 0; j < NJ; j++) { ex[j][0] = 0; ex[j][1] = 0; ex[j][2] = 0; ex[j][3] = 0; }
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const int8_t *nrow = p.ntt_rows + ((int64_t)k * p.vocab + ((cw >> (8 * (k + 1))) & 0xFF)) * H;
#pragma unroll
                    for (int j = 0; j < NJ; j++) {
                        const int32_t w4 = *reinterpret_cast<const int32_t *>(nrow + (j << 7) + (lane << 2));
#pragma unroll
                        for (int i = 0; i < 4; i++) ex[j][i] += (int)byte_of(w4, i) >> 2;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int32_t e4 = e4c[j];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    int prod = a_tok * (int)byte_of(emb_nb[j], i);
                    if (p.ov_emb_col) {
                        // (AccumType)(a_tok * b_dim * s_emb_row * s_emb_col), d-eggs kernels.cu:150-158: two float
                        // multiplications, each rounded, then the truncating conversion
                        const float fc = __fdiv_rn((float)overlay_num(byte_of(emb_oc[j], i)), 64.0f);
                        prod = __float2int_rz(__fmul_rn(__fmul_rn((float)prod, f_row), fc));
                    }
                    int perturb = (prod * ns) >> p.emb_shift;
                    x[j][i] = clip8((int)byte_of(e4, i) + emb_add[j][i] + perturb + (NTT ? ex[j][i] : 0));
                }
            }
        } else if (MODE == 2) {
            // the residual stream was requantised by the projection that produced it: only read it
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const uint32_t w = xw_next[j];
                xw_cur[j] = w;
                x[j][0] = ptx::sx_byte0(w); x[j][1] = ptx::sx_byte1(w); x[j][2] = ptx::sx_byte2(w); x[j][3] = (int)w >> 24;
            }
            if (r + 1 < r_end) {
#pragma unroll
                for (int j = 0; j < NJ; j++) xw_next[j] = *reinterpret_cast<const uint32_t *>(p.x_out + (int64_t)(r + 1) * H + (j << 7) + (lane << 2));
            }
        } else {
            int4 v[NJ];
#pragma unroll
            for (int j = 0; j < NJ; j++) v[j] = *reinterpret_cast<const int4 *>(p.pre32 + (int64_t)r * H + (j << 7) + (lane << 2));
            const int mx = p.rowmax[r];
            const float scale = aln_scale24(mx);
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                x[j][0] = aln_quant(v[j].x, scale); x[j][1] = aln_quant(v[j].y, scale);
                x[j][2] = aln_quant(v[j].z, scale); x[j][3] = aln_quant(v[j].w, scale);
            }
        }
        int tot = 0;
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int d = (j << 7) + (lane << 2);
            uint32_t w;
            if (MODE == 2) {
                w = xw_cur[j];                                                       // the bytes as they were read
            } else {
                w = ptx::pack_sat_s8(x[j][0], x[j][1], x[j][2], x[j][3]);            // |x| <= 127: the saturating pack is exact, two instructions
                *reinterpret_cast<uint32_t *>(p.x_out + (int64_t)r * H + d) = w;
            }
            tot = abs_sum4(w, tot);
        }
        // mean-abs norm with perturbed gain / bias (mgpu.cu:646-678): y = clip((x*w')/mn + b')
        tot = warp_sum(tot);
        int mn = tot / H;
        if (!mn) mn = 1;
        const float rinv = c_rinv_up.v[mn];                     // mn <= 127: a mean of absolute values of int8
        int dot[NDOTS];
#pragma unroll
        for (int q = 0; q < NDOTS; q++) dot[q] = 0;
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            const int d = (j << 7) + (lane << 2);
            int y[4];
#pragma unroll
            for (int i = 0; i < 4; i++) y[i] = div_small(x[j][i] * wv[j][i], rinv) * p.one + bv[j][i];   // the add as a multiply-add by a run-time 1: off the busier integer pipe
            const uint32_t yw = pack_clip8(y[0], y[1], y[2], y[3]);
            *reinterpret_cast<uint32_t *>(p.h_out + (int64_t)r * H + d) = yw;
#pragma unroll
            for (int q = 0; q < NDOTS; q++) dot[q] = __dp4a((int)yw, n4[q][j], dot[q]);
        }
#pragma unroll
        for (int q = 0; q < NDOTS; q++) {
            const int s = warp_sum(dot[q]);
            if (lane == 0) p.xb_out[(int64_t)r * p.xb_stride + q] = s;
        }
        if (lane == 0) {
            if (MODE == 1) p.rowmax[r] = 0;
            if (p.zero1) p.zero1[r] = 0;
            if (p.zero2) p.zero2[r] = 0;
            if (p.zero3) { p.zero3[(int64_t)r * 3] = 0; p.zero3[(int64_t)r * 3 + 1] = 0; p.zero3[(int64_t)r * 3 + 2] = 0; }
        }
    }
}

template <int MODE, int NDOTS, bool WIDE = false, bool NTT = false>
static int launch_rowwise_nj(cudaStream_t st, const RowParams &p) {
    const int blocks = ((p.M + ROW_RUN - 1) / ROW_RUN + 7) / 8;       // 8 warps per block, one run of rows per warp
    switch (p.H >> 7) {
        case 1: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 1, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        case 2: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 2, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        case 3: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 3, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        case 4: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 4, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        case 5: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 5, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        case 6: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 6, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        case 7: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 7, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        case 8: EGG_CUDA(launch_chained(rowwise_kernel<MODE, 8, NDOTS, WIDE, NTT>, blocks, 256, 0, st, p)); break;
        default: set_error("hidden_dim %d unsupported by the row-wise kernel", p.H); return EGG_E_INVALID;
    }
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

int launch_rowwise(cudaStream_t st, const RowParams &p_in, int mode) {
    RowParams p = p_in;
    p.fd_seq = make_fastdiv(p.seq_len);
    p.one = 1;
    if (p.ndots != 1 && p.ndots != 3) { set_error("row-wise kernel computes one or three row dots, not %d", p.ndots); return EGG_E_INVALID; }
    if (mode == 0 && (p.tok_wide || p.ntt_coef)) {
        if (p.ndots != 1 || p.vocab > 65536) { set_error("wide-token / transformed-window embedding takes one row dot and a vocabulary of at most 65536"); return EGG_E_INVALID; }
        if (p.ntt_coef) return p.tok_wide ? launch_rowwise_nj<0, 1, true, true>(st, p) : launch_rowwise_nj<0, 1, false, true>(st, p);
        return launch_rowwise_nj<0, 1, true>(st, p);
    }
    if (p.ndots == 1) return mode == 0 ? launch_rowwise_nj<0, 1>(st, p) : (mode == 1 ? launch_rowwise_nj<1, 1>(st, p) : launch_rowwise_nj<2, 1>(st, p));
    return mode == 0 ? launch_rowwise_nj<0, 3>(st, p) : (mode == 1 ? launch_rowwise_nj<1, 3>(st, p) : launch_rowwise_nj<2, 3>(st, p));
}

// Row dots under adaptive-noise overlays (d-eggs/include/model/layers.cuh:250, 272-280, 339-341, 396):
//   out[r][q] = Σ_tid pb(tid),  pb = 0;  for sub < terms:  pb = (int)((float)pb + x[k] * noise_q[k] * factor_q[k]),
//   k = tid + sub*H
// — with one term per thread this truncates every product, with four (the down projection) it truncates
// the thread's running sum.  All values are multiples of 1/64 below 2^17, so the float arithmetic of the
// reference is exact and is done here in integers: pb = trunc((64*pb + x*n*num) / 64).
//
// One warp per run of 8 rows of one member: noise times overlay numerator is the member's alone, formed once per run and kept
// as int16 pairs (|45 * 64| < 2^12); a product is then one two-term dot product against the word with its other byte masked.
// Bound: the integer pipe, about six instructions per product; at H 1024, 512 members x 512 tokens 434 -> 118 us on average.
constexpr int SDOT_RUN = 8;

template <int NJ, int TERMS, int NDOTS>
__global__ void __launch_bounds__(256) scaled_dot_kernel(const ScaledDotParams p) {
    chain_next();
    chain_wait();
    const int run = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    const int r0 = run * SDOT_RUN;
    if (r0 >= p.M) return;
    constexpr int H = NJ * 128, K = H * TERMS;
    const int mem = fast_div(r0, p.fd_seq);
    const int8_t *ntp = p.nt + (int64_t)(mem >> 1) * p.nt_stride;
    int32_t c[NDOTS][TERMS][NJ][2];
#pragma unroll
    for (int q = 0; q < NDOTS; q++)
#pragma unroll
        for (int t = 0; t < TERMS; t++)
#pragma unroll
            for (int j = 0; j < NJ; j++) {
                const int k = t * H + j * 128 + 4 * lane;
                const int32_t n4 = *reinterpret_cast<const int32_t *>(ntp + p.nt_dot[q] + k), o4 = *reinterpret_cast<const int32_t *>(p.ov[q] + k);
                int v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = (int)byte_of(n4, i) * overlay_num(byte_of(o4, i));
                c[q][t][j][0] = (v[0] & 0xFFFF) | (v[1] << 16);
                c[q][t][j][1] = (v[2] & 0xFFFF) | (v[3] << 16);
            }
    const int r1 = min(r0 + SDOT_RUN, p.M);
    for (int r = r0; r < r1; r++) {
        const int8_t *xr = p.x + (int64_t)r * K + 4 * lane;
        int acc[NDOTS] = {};
#pragma unroll
        for (int j = 0; j < NJ; j++) {
            int32_t x[TERMS];
#pragma unroll
            for (int t = 0; t < TERMS; t++) x[t] = *reinterpret_cast<const int32_t *>(xr + t * H + j * 128);
#pragma unroll
            for (int q = 0; q < NDOTS; q++) {
                int pb[4] = {0, 0, 0, 0};
#pragma unroll
                for (int t = 0; t < TERMS; t++) {
                    const int v0 = __dp2a_lo(c[q][t][j][0], x[t] & 0x000000FF, t ? pb[0] << 6 : 0), v1 = __dp2a_lo(c[q][t][j][0], x[t] & 0x0000FF00, t ? pb[1] << 6 : 0);
                    const int v2 = __dp2a_hi(c[q][t][j][1], x[t] & 0x00FF0000, t ? pb[2] << 6 : 0), v3 = __dp2a_hi(c[q][t][j][1], x[t] & (int)0xFF000000, t ? pb[3] << 6 : 0);
                    pb[0] = v0 / 64; pb[1] = v1 / 64; pb[2] = v2 / 64; pb[3] = v3 / 64;
                }
                acc[q] += pb[0] + pb[1] + pb[2] + pb[3];
            }
        }
#pragma unroll
        for (int q = 0; q < NDOTS; q++) {
            acc[q] = __reduce_add_sync(0xFFFFFFFFu, acc[q]);
            if (lane == 0) p.out[(int64_t)r * p.out_stride + q] = acc[q];
        }
    }
}

template <int TERMS, int NDOTS>
static int launch_scaled_dot_nj(cudaStream_t st, const ScaledDotParams &p) {
    const unsigned blocks = (unsigned)(((p.M + SDOT_RUN - 1) / SDOT_RUN + 7) / 8);
    switch (p.H >> 7) {
        case 1: EGG_CUDA(launch_chained(scaled_dot_kernel<1, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        case 2: EGG_CUDA(launch_chained(scaled_dot_kernel<2, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        case 3: EGG_CUDA(launch_chained(scaled_dot_kernel<3, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        case 4: EGG_CUDA(launch_chained(scaled_dot_kernel<4, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        case 5: EGG_CUDA(launch_chained(scaled_dot_kernel<5, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        case 6: EGG_CUDA(launch_chained(scaled_dot_kernel<6, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        case 7: EGG_CUDA(launch_chained(scaled_dot_kernel<7, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        case 8: EGG_CUDA(launch_chained(scaled_dot_kernel<8, TERMS, NDOTS>, blocks, 256, 0, st, p)); break;
        default: set_error("hidden_dim %d unsupported by the scaled row dots", p.H); return EGG_E_INVALID;
    }
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

int launch_scaled_dot(cudaStream_t st, const ScaledDotParams &p_in) {
    ScaledDotParams p = p_in;
    p.fd_seq = make_fastdiv(p.seq_len);
    if (p.terms == 4 && p.ndots == 1) return launch_scaled_dot_nj<4, 1>(st, p);
    if (p.terms == 1 && p.ndots == 1) return launch_scaled_dot_nj<1, 1>(st, p);
    if (p.terms == 1 && p.ndots == 3) return launch_scaled_dot_nj<1, 3>(st, p);
    set_error("scaled row dots: %d terms, %d dots unsupported", p.terms, p.ndots);
    return EGG_E_INVALID;
}

// Q/K/V requantisation (adaptive_qkv_normalize, mgpu.cu:782-784).  One warp per row; all of the row's loads
// (three parts x NJ 16-byte pieces per lane) are issued before any arithmetic.
template <int NJ>
__global__ void __launch_bounds__(256) aqn_kernel(const AqnParams p) {
    chain_next();
    chain_wait();
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= p.M) return;
    constexpr int H = NJ * 128;
    const int32_t *src = p.pre3 + (int64_t)r * 3 * H + (lane << 2);
    int4 v[3][NJ];
#pragma unroll
    for (int which = 0; which < 3; which++)
#pragma unroll
        for (int j = 0; j < NJ; j++) v[which][j] = *reinterpret_cast<const int4 *>(src + which * H + (j << 7));
    const int mx0 = p.rowmax3[(int64_t)r * 3], mx1 = p.rowmax3[(int64_t)r * 3 + 1], mx2 = p.rowmax3[(int64_t)r * 3 + 2];
#pragma unroll
    for (int which = 0; which < 3; which++) {
        const int mx = which == 0 ? mx0 : (which == 1 ? mx1 : mx2);
        const float scale = aln_scale24(mx);
        int8_t *out = (which == 0 ? p.q : (which == 1 ? p.k : p.v)) + (int64_t)r * H + (lane << 2);
#pragma unroll
        for (int j = 0; j < NJ; j++)
            *reinterpret_cast<uint32_t *>(out + (j << 7)) = pack_clip8(aln_quant(v[which][j].x, scale), aln_quant(v[which][j].y, scale),
                                                                       aln_quant(v[which][j].z, scale), aln_quant(v[which][j].w, scale));
    }
}

int launch_aqn(cudaStream_t st, const AqnParams &p) {
    const int blocks = (p.M + 7) / 8;
    switch (p.H >> 7) {
        case 1: EGG_CUDA(launch_chained(aqn_kernel<1>, blocks, 256, 0, st, p)); break;
        case 2: EGG_CUDA(launch_chained(aqn_kernel<2>, blocks, 256, 0, st, p)); break;
        case 3: EGG_CUDA(launch_chained(aqn_kernel<3>, blocks, 256, 0, st, p)); break;
        case 4: EGG_CUDA(launch_chained(aqn_kernel<4>, blocks, 256, 0, st, p)); break;
        case 5: EGG_CUDA(launch_chained(aqn_kernel<5>, blocks, 256, 0, st, p)); break;
        case 6: EGG_CUDA(launch_chained(aqn_kernel<6>, blocks, 256, 0, st, p)); break;
        case 7: EGG_CUDA(launch_chained(aqn_kernel<7>, blocks, 256, 0, st, p)); break;
        case 8: EGG_CUDA(launch_chained(aqn_kernel<8>, blocks, 256, 0, st, p)); break;
        default: set_error("hidden_dim %d unsupported by the requantisation kernel", p.H); return EGG_E_INVALID;
    }
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// =========================================================================
// causal integer-softmax attention (mgpu.cu:787-825), one block per (member, head)
// =========================================================================
// Scores and weighted sums run on the int8 tensor-core path (mma.sync m16n8k32):
// exact, because every partial sum is proven to fit int32 — scores <= 64*127^2,
// and the 19-bit softmax weights are split into three 7-bit limbs so that each
// limb's Σ w·v <= 127*127*seq_len; the limbs are recombined in int64 before the
// reference's truncating division.

__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the same product started from a zero accumulator: the outputs are written, not read, so no register has to be
// cleared first
__device__ __forceinline__ void mma_s8_first(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

// The same with the remainder assembled limb by limb; d0..d2 are the limb sums of the denominator.
__device__ __forceinline__ int att_div_limbs(int p0, int p1, int p2, int d0, int d1, int d2, float rden) {
    const float fn = fmaf(__int2float_rn(p2 * 128 + p1), 128.0f, __int2float_rn(p0));
    int k = __float2int_rn(fn * rden);
    const int r = (p0 - k * d0) + (p1 - k * d1) * 128 + (p2 - k * d2) * 16384;
    if (k > 0 && r < 0) k--;
    else if (k < 0 && r > 0) k++;
    return k;
}

// Layouts.  The contraction over the 64 head dims may run in any order as long as both operands agree, so lane q of a fragment
// takes dims 16q..16q+15: a query row is one 16-byte load, a key row one 16-byte shared read (64-byte pitch, conflict-free).
// The output columns may be dealt to tiles in any order too: tile dn holds dims 16(n>>1) + 2 dn + (n&1) in column n, so that a
// lane ends with 16 consecutive dims of its two rows: one 16-byte store each, and the noise dot on packed words.
constexpr int ATT_KP = 64;
__host__ __device__ __forceinline__ int att_vp(int SP) { return SP + (SP % 64 == 0 ? 32 : 0); }      // 32 modulo 64: 8-byte reads of four rows tile the banks

// scores of one 16-query x 32-key block: c[nt][0..3] for the four 8-key n-tiles
__device__ __forceinline__ void att_scores(int (&c)[4][4], const int4 (&qa)[2], const int8_t *Ks, int kb, int g, int q) {
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
        const int4 k = *reinterpret_cast<const int4 *>(Ks + (kb * 32 + nt * 8 + g) * ATT_KP + 16 * q);
        mma_s8_first(c[nt], qa[0].x, qa[1].x, qa[0].y, qa[1].y, k.x, k.y);
        mma_s8(c[nt], qa[0].z, qa[1].z, qa[0].w, qa[1].w, k.z, k.w);
    }
}

// trunc(num / den) as C does, for |num/den| <= 127: the quotient is estimated in float from the three
// limb sums and fixed up with one exact int64 remainder test.  (Limb sums below 2^23: att_div_small.)
__device__ __forceinline__ int att_div(int p0, int p1, int p2, long long den, float rden) {
    const long long num = (long long)p0 + ((long long)p1 << 7) + ((long long)p2 << 14);
    int k = f2i_exact((float)num * rden);             // nearest integer to the real quotient (|error| < 1e-3)
    long long r = num - (long long)k * den;
    if (num >= 0) { if (r < 0) k--; } else { if (r > 0) k++; }
    return k;
}

// limb-packed weights of a block's 16 scores per lane; keys beyond the query's own position weigh nothing
__device__ __forceinline__ void att_weights(uint32_t (&w)[4][4], const int (&c)[4][4], const uint32_t *lut3, int mxs0, int mxs1, int sh, bool masked, int key0,
                                            int row0, int row1) {
    // (a masked key may score above the maximum of the others: its index is not looked at)
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
        const int key = key0 + nt * 8;
        w[nt][0] = (!masked || key <= row0) ? lut3[min(255, mxs0 - (c[nt][0] >> sh))] : 0u;
        w[nt][1] = (!masked || key + 1 <= row0) ? lut3[min(255, mxs0 - (c[nt][1] >> sh))] : 0u;
        w[nt][2] = (!masked || key <= row1) ? lut3[min(255, mxs1 - (c[nt][2] >> sh))] : 0u;
        w[nt][3] = (!masked || key + 1 <= row1) ? lut3[min(255, mxs1 - (c[nt][3] >> sh))] : 0u;
    }
}
// A fragments of the three limbs; k-slot 4q+{0,1,2,3} <-> keys {2q, 2q+1, 8+2q, 9+2q} (+16 for registers 2, 3); limb sums of Σw
__device__ __forceinline__ void att_limbs(uint32_t (&al)[3][4], const uint32_t (&w)[4][4], int (&tl0)[3], int (&tl1)[3]) {
#pragma unroll
    for (int f = 0; f < 4; f++) {
        // 4 x 3 byte transpose of the four weights of fragment register f (7 byte permutes)
        const int n0 = (f >> 1) * 2, i0 = (f & 1) * 2;
        const uint32_t wa = w[n0][i0], wb = w[n0][i0 + 1], wc = w[n0 + 1][i0], wd = w[n0 + 1][i0 + 1];
        const uint32_t t0 = __byte_perm(wa, wb, 0x5140), t1 = __byte_perm(wc, wd, 0x5140);     // [a0 b0 a1 b1], [c0 d0 c1 d1]
        const uint32_t t2 = __byte_perm(wa, wb, 0x7362), t3 = __byte_perm(wc, wd, 0x7362);     // [a2 b2 . .], [c2 d2 . .]
        al[0][f] = __byte_perm(t0, t1, 0x5410);
        al[1][f] = __byte_perm(t0, t1, 0x7632);
        al[2][f] = __byte_perm(t2, t3, 0x5410);
    }
#pragma unroll
    for (int l = 0; l < 3; l++) {
        tl0[l] = __dp4a((int)al[l][0], 0x01010101, __dp4a((int)al[l][2], 0x01010101, tl0[l]));
        tl1[l] = __dp4a((int)al[l][1], 0x01010101, __dp4a((int)al[l][3], 0x01010101, tl1[l]));
    }
}
__device__ __forceinline__ int att_max(const int (&c)[4][4], int i, int mx) {
#pragma unroll
    for (int nt = 0; nt < 4; nt++) mx = max(mx, max(c[nt][i], c[nt][i + 1]));
    return mx;
}
__device__ __forceinline__ void att_max_masked(const int (&c)[4][4], int key0, int row0, int row1, int &mx0, int &mx1) {
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
        const int key = key0 + nt * 8;
        if (key <= row0) mx0 = max(mx0, c[nt][0]);
        if (key + 1 <= row0) mx0 = max(mx0, c[nt][1]);
        if (key <= row1) mx1 = max(mx1, c[nt][2]);
        if (key + 1 <= row1) mx1 = max(mx1, c[nt][3]);
    }
}
__device__ __forceinline__ int quad_max(int v) {
    v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, 1));
    return max(v, __shfl_xor_sync(0xFFFFFFFFu, v, 2));
}
__device__ __forceinline__ int quad_sum(int v) {
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    return v + __shfl_xor_sync(0xFFFFFFFFu, v, 2);
}

// Quotients of tile dn (rows g and g+8, two dims each) into the packed output words.
struct AttOut { uint32_t w0[4], w1[4]; };
// LONG: limbs of the denominators (tl0, tl1) instead of its low word -- more instructions, fewer registers live at the end of
// the long form, where the shorter chain measured 2.5 % slower.
template <bool LONG>
__device__ __forceinline__ void att_quotients(AttOut &o, int dn, const int (&acc)[3][4], const int (&tl0)[3], const int (&tl1)[3], long long den0, long long den1,
                                              float rden0, float rden1, bool small_limbs) {
    int v[4];
    if (small_limbs) {
        // |Σw·v / Σw| <= 127 (a weighted mean of int8 values): the reference's clip cannot trigger
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (LONG) v[i] = i < 2 ? att_div_limbs(acc[0][i], acc[1][i], acc[2][i], tl0[0], tl0[1], tl0[2], rden0)
                                   : att_div_limbs(acc[0][i], acc[1][i], acc[2][i], tl1[0], tl1[1], tl1[2], rden1);
            else v[i] = att_div_small(acc[0][i], acc[1][i], acc[2][i], (uint32_t)(i < 2 ? den0 : den1), i < 2 ? rden0 : rden1);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = clip8(att_div(acc[0][i], acc[1][i], acc[2][i], i < 2 ? den0 : den1, i < 2 ? rden0 : rden1));
    }
    if (dn & 1) {
        o.w0[dn >> 1] = __byte_perm(o.w0[dn >> 1], __byte_perm((uint32_t)v[0], (uint32_t)v[1], 0x0040), 0x5410);
        o.w1[dn >> 1] = __byte_perm(o.w1[dn >> 1], __byte_perm((uint32_t)v[2], (uint32_t)v[3], 0x0040), 0x5410);
    } else {
        o.w0[dn >> 1] = __byte_perm((uint32_t)v[0], (uint32_t)v[1], 0x0040);
        o.w1[dn >> 1] = __byte_perm((uint32_t)v[2], (uint32_t)v[3], 0x0040);
    }
}
__device__ __forceinline__ void att_store(const AttnParams &p, const AttOut &o, const int4 nb, int64_t row0, int col, int q) {
    *reinterpret_cast<uint4 *>(p.ao + row0 * p.H + col) = make_uint4(o.w0[0], o.w0[1], o.w0[2], o.w0[3]);
    *reinterpret_cast<uint4 *>(p.ao + (row0 + 8) * p.H + col) = make_uint4(o.w1[0], o.w1[1], o.w1[2], o.w1[3]);
    int d0 = __dp4a((int)o.w0[0], nb.x, __dp4a((int)o.w0[1], nb.y, __dp4a((int)o.w0[2], nb.z, __dp4a((int)o.w0[3], nb.w, 0))));
    int d1 = __dp4a((int)o.w1[0], nb.x, __dp4a((int)o.w1[1], nb.y, __dp4a((int)o.w1[2], nb.z, __dp4a((int)o.w1[3], nb.w, 0))));
    d0 = quad_sum(d0);
    d1 = quad_sum(d1);
    if (q == 0) {
        atomicAdd(&p.xbo[row0], d0);
        atomicAdd(&p.xbo[row0 + 8], d1);
    }
}

// One 16-query block of one head by one warp.  Ks, Vt: the head's keys and transposed values in shared memory.
// KB > 0: at most KB key blocks (seq_len <= 32 KB): the scores stay in registers between the maximum and the weights, all limb
// fragments are formed before the products, and an output tile is accumulated, divided and done (12 accumulators instead of 96).
// KB = 0: any length; scores are computed twice, all output tiles accumulate side by side.
template <int KB>
__device__ __forceinline__ void att_query_block(const AttnParams &p, const int8_t *Ks, const int8_t *Vt, const uint32_t *lut3, int VP, int64_t base, int col0,
                                                const int8_t *nbo, int qb, int lane, bool small_limbs) {
    const int H = p.H, g = lane >> 2, q = lane & 3, sh = p.shift_attn;
    const int q0 = qb * 16, row0 = q0 + g, row1 = row0 + 8, last = (q0 + 15) / 32;      // last: the only key block that needs the causal mask
    int4 qa[2];
    qa[0] = *reinterpret_cast<const int4 *>(p.q + (base + row0) * H + col0 + 16 * q);
    qa[1] = *reinterpret_cast<const int4 *>(p.q + (base + row1) * H + col0 + 16 * q);
    const int4 nb = *reinterpret_cast<const int4 *>(nbo + 16 * q);
    int mx0 = INT_MIN, mx1 = INT_MIN;
    int tl0[3] = {0, 0, 0}, tl1[3] = {0, 0, 0};              // per-limb Σw of rows g and g+8
    AttOut out;
    const int8_t *vb = Vt + g * VP + 8 * q;
    if (KB > 0) {
        constexpr int NB = KB > 0 ? KB : 1;
        int c[NB][4][4];
        uint32_t al[NB][3][4];
#pragma unroll
        for (int kb = 0; kb < NB; kb++) {
            if (kb > last) continue;
            att_scores(c[kb], qa, Ks, kb, g, q);
            if (kb < last) { mx0 = att_max(c[kb], 0, mx0); mx1 = att_max(c[kb], 2, mx1); }
            else att_max_masked(c[kb], kb * 32 + 2 * q, row0, row1, mx0, mx1);
        }
        mx0 = quad_max(mx0) >> sh;
        mx1 = quad_max(mx1) >> sh;
#pragma unroll
        for (int kb = 0; kb < NB; kb++) {
            if (kb > last) continue;
            uint32_t w[4][4];
            if (kb < last) att_weights(w, c[kb], lut3, mx0, mx1, sh, false, 0, row0, row1);
            else att_weights(w, c[kb], lut3, mx0, mx1, sh, true, kb * 32 + 2 * q, row0, row1);
            att_limbs(al[kb], w, tl0, tl1);
        }
#pragma unroll
        for (int l = 0; l < 3; l++) { tl0[l] = quad_sum(tl0[l]); tl1[l] = quad_sum(tl1[l]); }
        const uint32_t tot0 = (uint32_t)tl0[0] + ((uint32_t)tl0[1] << 7) + ((uint32_t)tl0[2] << 14);
        const uint32_t tot1 = (uint32_t)tl1[0] + ((uint32_t)tl1[1] << 7) + ((uint32_t)tl1[2] << 14);
        const uint32_t den0 = tot0 ? tot0 : 1, den1 = tot1 ? tot1 : 1;
        const float rden0 = 1.0f / (float)den0, rden1 = 1.0f / (float)den1;
#pragma unroll
        for (int dn = 0; dn < 8; dn++) {
            int acc[3][4];
#pragma unroll
            for (int kb = 0; kb < NB; kb++) {
                if (kb > last) continue;
                const int2 b = *reinterpret_cast<const int2 *>(vb + dn * 8 * VP + kb * 32);
#pragma unroll
                for (int l = 0; l < 3; l++) {
                    if (kb == 0) mma_s8_first(acc[l], al[0][l][0], al[0][l][1], al[0][l][2], al[0][l][3], b.x, b.y);
                    else mma_s8(acc[l], al[kb][l][0], al[kb][l][1], al[kb][l][2], al[kb][l][3], b.x, b.y);
                }
            }
            att_quotients<false>(out, dn, acc, tl0, tl1, den0, den1, rden0, rden1, true);
        }
    } else {
        int c[4][4];
        // ---- pass 1: row maxima over ctx <= t (mgpu.cu:795-802) ----
        for (int kb = 0; kb < last; kb++) {
            att_scores(c, qa, Ks, kb, g, q);
            mx0 = att_max(c, 0, mx0);
            mx1 = att_max(c, 2, mx1);
        }
        att_scores(c, qa, Ks, last, g, q);
        att_max_masked(c, last * 32 + 2 * q, row0, row1, mx0, mx1);
        mx0 = quad_max(mx0) >> sh;
        mx1 = quad_max(mx1) >> sh;
        // ---- pass 2: weights, Σ w·v in three 7-bit limbs (mgpu.cu:810-824) ----
        int acc[8][3][4];
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int l = 0; l < 3; l++)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[a][l][i] = 0;
        for (int kb = 0; kb <= last; kb++) {
            att_scores(c, qa, Ks, kb, g, q);
            uint32_t w[4][4], al[3][4];
            if (kb < last) att_weights(w, c, lut3, mx0, mx1, sh, false, 0, row0, row1);
            else att_weights(w, c, lut3, mx0, mx1, sh, true, kb * 32 + 2 * q, row0, row1);
            att_limbs(al, w, tl0, tl1);
#pragma unroll
            for (int dn = 0; dn < 8; dn++) {
                const int2 b = *reinterpret_cast<const int2 *>(vb + dn * 8 * VP + kb * 32);
#pragma unroll
                for (int l = 0; l < 3; l++) mma_s8(acc[dn][l], al[l][0], al[l][1], al[l][2], al[l][3], b.x, b.y);
            }
        }
#pragma unroll
        for (int l = 0; l < 3; l++) { tl0[l] = quad_sum(tl0[l]); tl1[l] = quad_sum(tl1[l]); }
        const uint32_t tot0 = (uint32_t)tl0[0] + ((uint32_t)tl0[1] << 7) + ((uint32_t)tl0[2] << 14);
        const uint32_t tot1 = (uint32_t)tl1[0] + ((uint32_t)tl1[1] << 7) + ((uint32_t)tl1[2] << 14);
        const long long den0 = tot0 ? (long long)tot0 : 1, den1 = tot1 ? (long long)tot1 : 1;
        const float rden0 = 1.0f / (float)den0, rden1 = 1.0f / (float)den1;
#pragma unroll
        for (int dn = 0; dn < 8; dn++) att_quotients<true>(out, dn, acc[dn], tl0, tl1, den0, den1, rden0, rden1, small_limbs);
    }
    att_store(p, out, nb, base + row0, col0 + 16 * q, q);
}

// Keys and transposed values of one head into shared memory by `nt` threads (this one is number `t`).
__device__ __forceinline__ void att_stage(const AttnParams &p, int8_t *Ks, int8_t *Vt, int SP, int VP, int64_t base, int col0, int t, int nt) {
    const int S = p.seq_len, H = p.H;
    for (int i = t; i < SP * 4; i += nt) {
        const int row = i >> 2, ch = i & 3;
        int4 v = make_int4(0, 0, 0, 0);
        if (row < S) v = *reinterpret_cast<const int4 *>(p.k + (base + row) * H + col0 + ch * 16);
        *reinterpret_cast<int4 *>(Ks + row * ATT_KP + ch * 16) = v;
    }
    // V: each item = 4 consecutive keys x 16 dims, transposed in registers (4x4 byte blocks).  Row r of Vt is output column
    // r & 7 of tile r >> 3; inside a row the keys of a 32-block are ordered so that the two registers of a fragment are one
    // 8-byte word: keys {2q, 2q+1, 8+2q, 9+2q} at 8q, the same + 16 at 8q + 4.
    for (int i = t; i < (SP / 4) * 4; i += nt) {
        const int kg = i % (SP / 4), ch = i / (SP / 4);
        int4 r[4];
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            const int row = kg * 4 + kk;
            r[kk] = make_int4(0, 0, 0, 0);
            if (row < S) r[kk] = *reinterpret_cast<const int4 *>(p.v + (base + row) * H + col0 + ch * 16);
        }
        const uint32_t *w0 = reinterpret_cast<const uint32_t *>(&r[0]), *w1 = reinterpret_cast<const uint32_t *>(&r[1]);
        const uint32_t *w2 = reinterpret_cast<const uint32_t *>(&r[2]), *w3 = reinterpret_cast<const uint32_t *>(&r[3]);
        const int m = kg & 3;
        const int so = (kg >> 3) * 32 + ((m & 1) * 2) * 8 + ((kg >> 2) & 1) * 4 + (m >> 1) * 2;     // keys 4m, 4m+1; keys 4m+2, 4m+3 eight further
#pragma unroll
        for (int dq = 0; dq < 4; dq++) {       // dims 4dq..4dq+3 of this chunk
            const uint32_t p0 = __byte_perm(w0[dq], w1[dq], 0x5140), p1 = __byte_perm(w2[dq], w3[dq], 0x5140);   // [a0 b0 a1 b1]
            const uint32_t p2 = __byte_perm(w0[dq], w1[dq], 0x7362), p3 = __byte_perm(w2[dq], w3[dq], 0x7362);   // [a2 b2 a3 b3]
            uint32_t d[4];
            d[0] = __byte_perm(p0, p1, 0x5410); d[1] = __byte_perm(p0, p1, 0x7632);
            d[2] = __byte_perm(p2, p3, 0x5410); d[3] = __byte_perm(p2, p3, 0x7632);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int dl = dq * 4 + j;     // dim 16 ch + dl: tile dl >> 1, column 2 ch + (dl & 1)
                int8_t *o = Vt + ((dl >> 1) * 8 + 2 * ch + (dl & 1)) * VP + so;
                *reinterpret_cast<uint16_t *>(o) = (uint16_t)d[j];
                *reinterpret_cast<uint16_t *>(o + 8) = (uint16_t)(d[j] >> 16);
            }
        }
    }
}

__device__ __forceinline__ void att_table(uint32_t *lut3, const int32_t *exp_lut, int t, int nt) {
    for (int i = t; i < 256; i += nt) {
        const uint32_t w = (uint32_t)exp_lut[i];
        lut3[i] = (w & 127u) | (((w >> 7) & 127u) << 8) | ((w >> 14) << 16);
    }
}

// One block per head.  KB = 0: any length (168 registers, three blocks per SM); KB = 4: up to 128 tokens.
template <int KB>
__global__ void __launch_bounds__(128, 3) attention_kernel(const AttnParams p) {
    chain_next();
    chain_wait();
    extern __shared__ __align__(16) uint8_t att_smem[];
    const int S = p.seq_len, SP = (S + 31) & ~31, VP = att_vp(SP), H = p.H;
    int8_t *Ks = reinterpret_cast<int8_t *>(att_smem);          // [SP][64]
    int8_t *Vt = Ks + SP * ATT_KP;                               // [64][VP]
    uint32_t *lut3 = reinterpret_cast<uint32_t *>(Vt + 64 * VP); // [256] softmax weight as three 7-bit limbs, one per byte
    const int n_heads = H / 64;
    const int mem = blockIdx.x / n_heads, hd = blockIdx.x % n_heads;
    const int64_t base = (int64_t)mem * p.row_stride;
    const int col0 = hd * 64;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    att_stage(p, Ks, Vt, SP, VP, base, col0, tid, 128);
    att_table(lut3, p.exp_lut, tid, 128);
    __syncthreads();
    const int8_t *nbo = p.nt + (int64_t)(mem >> 1) * p.nt_stride + p.nt_o_b + col0;
    // Query blocks are dealt to the four warps in boustrophedon order (w, 7-w, 8+w, 15-w, ...): block qb costs
    // qb/2 + 1 key blocks under the causal mask, and this order gives every warp the same total (18 of 72 at
    // seq_len 256) where the plain stride-4 order leaves warp 3 with 20 and warp 0 with 16.
    for (int rnd = 0; rnd * 4 < S / 16; rnd++) {
        const int qb = rnd * 4 + ((rnd & 1) ? 3 - warp : warp);
        if (qb >= S / 16) continue;
        att_query_block<KB>(p, Ks, Vt, lut3, VP, base, col0, nbo, qb, lane, S <= 512);     // limb sums below 127*127*512 < 2^23
    }
}

// Short sequences: a warp per head, on its own from loading to storing.  With a block per head, seq_len 32 is two query blocks
// for four warps behind one barrier, and the block's latency is all there is.
template <int KB>
__global__ void __launch_bounds__(128) attention_warp_kernel(const AttnParams p) {
    chain_next();
    chain_wait();
    extern __shared__ __align__(16) uint8_t att_smem[];
    const int S = p.seq_len, SP = KB * 32, VP = att_vp(SP), H = p.H, n_heads = H / 64;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *lut3 = reinterpret_cast<uint32_t *>(att_smem);
    int8_t *Ks = reinterpret_cast<int8_t *>(att_smem + 1024) + warp * (SP * ATT_KP + 64 * VP), *Vt = Ks + SP * ATT_KP;
    att_table(lut3, p.exp_lut, threadIdx.x, 128);
    __syncthreads();
    const int item = (int)blockIdx.x * 4 + warp;
    if (item >= p.members * n_heads) return;
    const int mem = item / n_heads, col0 = (item % n_heads) * 64;
    const int64_t base = (int64_t)mem * p.row_stride;
    att_stage(p, Ks, Vt, SP, VP, base, col0, lane, 32);
    __syncwarp();
    const int8_t *nbo = p.nt + (int64_t)(mem >> 1) * p.nt_stride + p.nt_o_b + col0;
#pragma unroll 1
    for (int qb = 0; qb < S / 16; qb++) att_query_block<KB>(p, Ks, Vt, lut3, VP, base, col0, nbo, qb, lane, true);
}

static size_t attention_smem_bytes(int SP, int heads) { return (size_t)heads * (SP * ATT_KP + 64 * (size_t)att_vp(SP)) + 256 * 4; }

template <typename F>
static int launch_attention_form(cudaStream_t st, F kern, int form, unsigned blocks, size_t smem, const AttnParams &p) {
    static std::atomic<bool> configured[4][EGG_MAX_DEVICES] = {};
    EGG_CUDA(allow_all_smem(kern, configured[form]));
    EGG_CUDA(launch_chained(kern, blocks, 128, smem, st, p));
    return EGG_OK;
}

int launch_attention(cudaStream_t st, const AttnParams &p) {
    const int heads = p.members * (p.H / 64), SP = (p.seq_len + 31) & ~31;
    // up to 64 tokens a warp takes a head; up to 128 four warps share one and keep their scores in registers
    if (p.seq_len <= 32) return launch_attention_form(st, attention_warp_kernel<1>, 0, (unsigned)((heads + 3) / 4), attention_smem_bytes(32, 4), p);
    if (p.seq_len <= 64) return launch_attention_form(st, attention_warp_kernel<2>, 1, (unsigned)((heads + 3) / 4), attention_smem_bytes(64, 4), p);
    if (p.seq_len <= 128) return launch_attention_form(st, attention_kernel<4>, 2, (unsigned)heads, attention_smem_bytes(SP, 1), p);
    return launch_attention_form(st, attention_kernel<0>, 3, (unsigned)heads, attention_smem_bytes(SP, 1), p);
}

// =========================================================================
// weights: packed [K/4][N][4] -> K-major shadow [N][K]
// =========================================================================
__global__ void unpack_transpose_kernel(const int32_t *packed, int8_t *shadow, int rows_k, int cols_n) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t words = (int64_t)(rows_k >> 2) * cols_n;
    if (i >= words) return;
    // consecutive threads take consecutive k4 of one output column: 128-byte coalesced writes
    int k4 = (int)(i % (rows_k >> 2));
    int n = (int)(i / (rows_k >> 2));
    int32_t w = packed[(int64_t)k4 * cols_n + n];
    *reinterpret_cast<int32_t *>(shadow + (int64_t)n * rows_k + 4 * k4) = w;
}

int launch_unpack_transpose(cudaStream_t st, const int8_t *packed, int8_t *shadow, int rows_k, int cols_n) {
    int64_t words = (int64_t)(rows_k >> 2) * cols_n;
    unpack_transpose_kernel<<<(unsigned)((words + 255) / 256), 256, 0, st>>>(reinterpret_cast<const int32_t *>(packed), shadow, rows_k, cols_n);
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// =========================================================================
// transform of each pair's input window (NTT_MODE 1..3; egg_ntt.cuh, called mgpu.cu:877-887): one block per pair,
// the window in shared memory.  Mode 1: Walsh-Hadamard butterflies (a, b) -> (a + b, a - b) over strides 1, 2, 4, ...
// Modes 2 / 3: values reduced mod p = 257 / 65537, bit-reversal, then log2(len) decimation-in-time stages whose
// twiddle is 3^(j * len / m) mod p -- the reference takes the root of the full-length transform whatever len is.
// Both members of a pair read the same window, so the coefficients are kept per pair.
// =========================================================================
__device__ __forceinline__ uint32_t fermat_pow3(uint32_t prime, int k) {
    k &= (int)(prime - 2);                 // prime - 1 is a power of two
    unsigned long long r = 1, b = 3;
    while (k > 0) {
        if (k & 1) r = r * b % prime;
        b = b * b % prime;
        k >>= 1;
    }
    return (uint32_t)r;
}

__global__ void __launch_bounds__(512) window_transform_kernel(const WindowParams p) {
    chain_next();
    chain_wait();
    extern __shared__ int32_t s_win[];
    const int S = p.seq_len, tid = threadIdx.x;
    const int64_t pair = p.pair_base + blockIdx.x;
    const int64_t pos = p.use_same_data ? (p.start_idx % (p.data_len - S)) : ((p.start_idx + pair * p.data_stride) % (p.data_len - S));
    const uint32_t prime = p.mode == 2 ? 257u : 65537u;
    for (int i = tid; i < S; i += blockDim.x) {
        const uint32_t tok = p.tok_wide ? reinterpret_cast<const uint32_t *>(p.dataset)[pos + i] : (uint32_t)p.dataset[pos + i];
        s_win[i] = p.mode == 1 ? (int32_t)tok : (int32_t)(tok % prime);
    }
    __syncthreads();
    if (p.mode == 1) {
        for (int stride = 1; stride < S; stride <<= 1) {
            for (int t = tid; t < (S >> 1); t += blockDim.x) {
                const int base = (t / stride) * 2 * stride + (t % stride);
                const int32_t a = s_win[base], b = s_win[base + stride];
                s_win[base] = a + b; s_win[base + stride] = a - b;
            }
            __syncthreads();
        }
    } else {
        const int lg = 31 - __clz(S);
        for (int i = tid; i < S; i += blockDim.x) {
            const int rev = (int)(__brev((unsigned)i) >> (32 - lg));
            if (i < rev) { const int32_t t = s_win[i]; s_win[i] = s_win[rev]; s_win[rev] = t; }
        }
        __syncthreads();
        for (int s = 1; s <= lg; s++) {
            const int m2 = 1 << (s - 1), w_step = S >> s;
            for (int k = tid; k < (S >> 1); k += blockDim.x) {
                const int j = k & (m2 - 1), i1 = ((k >> (s - 1)) << s) + j, i2 = i1 + m2;
                const uint32_t wb = (uint32_t)((unsigned long long)fermat_pow3(prime, j * w_step) * (uint32_t)s_win[i2] % prime);
                const uint32_t a = (uint32_t)s_win[i1];
                s_win[i1] = (int32_t)((a + wb) % prime);
                s_win[i2] = (int32_t)((a + prime - wb) % prime);
            }
            __syncthreads();
        }
    }
    for (int i = tid; i < S; i += blockDim.x) p.coef[(int64_t)blockIdx.x * S + i] = s_win[i];
}
int launch_window_transform(cudaStream_t st, const WindowParams &p) {
    if (p.mode < 1 || p.mode > 3 || p.seq_len < 2 || (p.seq_len & (p.seq_len - 1)) || p.seq_len > 8192 || p.pairs <= 0) {
        set_error("window transform: mode %d, seq_len %d, %d pairs unsupported", p.mode, p.seq_len, p.pairs); return EGG_E_INVALID;
    }
    int threads = p.seq_len / 2 < 32 ? 32 : (p.seq_len / 2 > 512 ? 512 : p.seq_len / 2);
    EGG_CUDA(launch_chained(window_transform_kernel, p.pairs, threads, (size_t)p.seq_len * sizeof(int32_t), st, p));
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// =========================================================================
// cross-entropy over stored logits: second pass of the head when the vocabulary is wider than one GEMM tile
// (mgpu.cu:985-1023).  One warp per row: the row's maximum from the maxima of 64, Σ exp-table[max - logit] in 64 bits, the
// target's logit, then loss[member] += (log_sum >> 1) + max - target with log_sum = 16 * (floor(log2 Σ) - SOFTMAX_SCALE_BIT).
// Bound by shared-memory lookups, one per logit and lane: the table has a copy per bank and goes on with its last entry, so
// that (maximum - maximum of the 64) + byte indexes it without a minimum; 64 logits that are all 255 below need no bytes.
// =========================================================================
constexpr int HEAD_LOSS_THREADS = 512;
constexpr int HEAD_LOSS_SMEM = 512 * 32 * 4;
__global__ void __launch_bounds__(HEAD_LOSS_THREADS, 3) head_loss_kernel(const HeadLossParams p, uint32_t stride) {
    chain_next();
    extern __shared__ uint32_t s_lut[];            // [512][32]
    for (int i = threadIdx.x; i < 512 * 32; i += HEAD_LOSS_THREADS) s_lut[i] = (uint32_t)p.exp_lut[min(255, i >> 5)];
    __syncthreads();
    chain_wait();
    const int lane = threadIdx.x & 31;
    const uint32_t lut = ptx::smem_u32(s_lut) + 4 * lane;
    const uint32_t last = s_lut[255 * 32 + lane];
    const int groups = p.V >> 6;
    for (int r = blockIdx.x * (HEAD_LOSS_THREADS / 32) + (threadIdx.x >> 5); r < p.M; r += gridDim.x * (HEAD_LOSS_THREADS / 32)) {
        const int mem = fast_div(r, p.fd_seq), t = r - mem * p.seq_len;
        if (t >= p.tok_len) continue;
        const int32_t *gm = p.max64 + (int64_t)r * groups;
        int mx = INT_MIN;
        for (int g = lane; g < groups; g += 32) mx = max(mx, gm[g]);
        mx = __reduce_max_sync(0xFFFFFFFFu, mx);
        const uint8_t *row = p.below + (int64_t)r * p.V;
        unsigned long long sum = 0;
#pragma unroll 4
        for (int c = lane << 4; c < p.V; c += 512) {
            const int off = mx - gm[c >> 6];
            if (off >= 255) { sum += (unsigned long long)last * 16; continue; }
            const int4 b = __ldcs(reinterpret_cast<const int4 *>(row + c));            // read once
            const uint32_t w[4] = {(uint32_t)b.x, (uint32_t)b.y, (uint32_t)b.z, (uint32_t)b.w};
            const uint32_t base = lut + (uint32_t)off * stride;
            uint32_t part = 0;
#pragma unroll
            for (int k = 0; k < 4; k++)
                part += ptx::lds_u32(__dp4a(w[k], stride, base)) + ptx::lds_u32(__dp4a(w[k], stride << 8, base)) +
                        ptx::lds_u32(__dp4a(w[k], stride << 16, base)) + ptx::lds_u32(__dp4a(w[k], stride << 24, base));
            sum += part;                           // 16 entries of at most 2^softmax_scale_bit
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        // the target's logit: one row of the product once more (its byte may have saturated)
        const int64_t pair = (p.pop_base + mem) >> 1;
        const int64_t pos = p.use_same_data ? (p.start_idx % (p.data_len - p.tok_len))
                                            : ((p.start_idx + pair * p.data_stride) % (p.data_len - p.tok_len));
        const uint32_t target = p.dataset[pos + t + 1];
        int tgt = 0;                               // no column matches: s_target_logit stays 0
        if (target < (uint32_t)p.V) {
            int acc = 0;
            for (int k = lane << 2; k < p.H; k += 128)
                acc = __dp4a(*reinterpret_cast<const int32_t *>(p.h + (int64_t)r * p.H + k), *reinterpret_cast<const int32_t *>(p.emb + (int64_t)target * p.H + k), acc);
            acc = __reduce_add_sync(0xFFFFFFFFu, acc);
            const int xb = p.xb[(int64_t)r * p.xb_stride], a = p.nt[(int64_t)(mem >> 1) * p.nt_stride + p.nt_a_off + target];
            tgt = (acc + ((((mem & 1) ? -xb : xb) * a) >> p.rank1_shift)) >> p.out_shift;
        }
        if (lane == 0) {
            long long log_sum = 0;
            if (sum > 0) log_sum = ((long long)(63 - __clzll((long long)sum)) << 4) - ((long long)p.softmax_scale_bit << 4);   // shift ladder of mgpu.cu:1012-1019
            atomicAdd(&p.loss[mem], (int)((log_sum >> 1) + mx - tgt));
        }
    }
}
int launch_head_loss(cudaStream_t st, const HeadLossParams &p_in, int num_sms) {
    HeadLossParams p = p_in;
    if (p.M <= 0 || p.V % 256 || p.V <= 0 || p.H % 128) { set_error("head loss: unsupported shape M=%d V=%d H=%d", p.M, p.V, p.H); return EGG_E_INVALID; }
    p.fd_seq = make_fastdiv(p.seq_len);
    static bool attr_set[EGG_MAX_DEVICES] = {};
    bool &done = attr_set[current_device_slot()];
    if (!done) { EGG_CUDA(cudaFuncSetAttribute(head_loss_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, HEAD_LOSS_SMEM)); done = true; }
    const int want = (p.M + HEAD_LOSS_THREADS / 32 - 1) / (HEAD_LOSS_THREADS / 32);
    EGG_CUDA(launch_chained(head_loss_kernel, want < 3 * num_sms ? want : 3 * num_sms, HEAD_LOSS_THREADS, HEAD_LOSS_SMEM, st, p, 32u * 4));
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// =========================================================================
// fitness (mgpu.cu:1031-1036)
// =========================================================================
// copy: pinned host memory for the losses, or null (stores over PCIe that the update hides; a copy of its own cost 6 us at its end)
__global__ void fitness_kernel(const int32_t *loss, int32_t *fit, int pairs, int2 *copy) {
    chain_next();
    chain_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pairs) return;
    int32_t pz = loss[2 * i], n = loss[2 * i + 1];
    if (copy) copy[i] = make_int2(pz, n);
    fit[i] = (pz < n) ? 1 : ((n < pz) ? -1 : 0);
}
int launch_fitness(cudaStream_t st, const int32_t *loss, int32_t *fit, int pairs, int32_t *copy) {
    EGG_CUDA(launch_chained(fitness_kernel, (pairs + 255) / 256, 256, 0, st, loss, fit, pairs, reinterpret_cast<int2 *>(copy)));
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// 16 bytes into pinned host memory: a third of what a copy costs at the end of a chain of kernels
__global__ void publish_kernel(int4 *dst, const int4 *src) {
    chain_wait();
    *dst = *src;
}
int launch_publish(cudaStream_t st, void *dst, const void *src) {
    EGG_CUDA(launch_chained(publish_kernel, 1, 1, 0, st, static_cast<int4 *>(dst), static_cast<const int4 *>(src)));
    return EGG_OK;
}

// =========================================================================
// update operands: the two noise matrices of vote = Σ_p f_p a_p b_p^T, pair index contiguous
// =========================================================================
// The update kernels are bound by the integer pipe (half the rate of the multiply-add pipe): the single-field noise
// value's sign select and the seed additions are written as multiply-adds with run-time multipliers (constants would
// be folded back into integer-pipe instructions).  hash_mix(seed + idx * 0x9e3779b9) == hash_rng(seed, idx).
struct UpdMul { int one, two; };
static inline UpdMul make_upd_mul() { UpdMul m; m.one = 1; m.two = 2; return m; }
__device__ __forceinline__ uint32_t hash_mix(uint32_t x) {
    x ^= x >> 16; x *= 0x85ebca6bu;
    x ^= x >> 13; x *= 0xc2b2ae35u;
    x ^= x >> 16;
    return x;
}

constexpr int UPD_ROWS_PER_BLOCK = 8;     // operand rows one block writes: the pair seeds and fitness words are loaded once for all of them

template <bool GAUSS>
__global__ void __launch_bounds__(256) update_operands_kernel(int8_t *na, int8_t *nb, const int32_t *fit, int pairs, int kp, int rows_k, int cols_n,
                                       int off_a, int off_b, int seed_base, uint32_t step_seed, int mask, int split, const UpdMul um) {
    const int row0 = blockIdx.y * UPD_ROWS_PER_BLOCK;      // 0..cols_n-1 -> NA, cols_n.. -> NB (cols_n is a multiple of the group size)
    const int ktot = split ? 2 * kp : kp;
    const bool is_a = row0 < cols_n;
    // four consecutive pair slots per thread (kp is a multiple of 128): one word store per row, two when the contraction is split:
    // both halves hold the same noise, hashed once (4096 x 4096 over 32 768 pairs: 430 -> 240 us; the hashes are what it is bound by)
    for (int pp = (blockIdx.x * blockDim.x + threadIdx.x) * 4; pp < kp; pp += gridDim.x * blockDim.x * 4) {
        uint32_t seed[4];
        int f[4], fh[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int pidx = pp + j;
            seed[j] = step_seed + (uint32_t)pidx + (uint32_t)seed_base + (uint32_t)(is_a ? off_a : off_b);    // mgpu.cu:1095
            f[j] = 0; fh[j] = 0;                          // 0 for the padding beyond the last pair
            if (pidx < pairs) {
                f[j] = is_a ? fit[pidx] : 1; fh[j] = 16;
                if (is_a && split) { fh[j] = f[j] >> 4; f[j] -= fh[j] << 4; }
            }
        }
#pragma unroll
        for (int rr = 0; rr < UPD_ROWS_PER_BLOCK; rr++) {
            const int row = row0 + rr;
            const uint32_t idx = (uint32_t)(is_a ? row : row - cols_n);
            int val[4], vh[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (GAUSS) {
                    const int n = noise_from_hash(seed[j], idx, mask, 1);
                    val[j] = f[j] * n; vh[j] = fh[j] * n;
                } else {
                    // f * noise_field(r, 0, 1, mask): magnitude (r >> 1) & mask, positive when bit 0 is set
                    const uint32_t r = hash_mix(seed[j] * (uint32_t)um.one + idx * 0x9e3779b9u);
                    const int n = (int)((r >> 1) & (uint32_t)mask) * ((int)(r & 1u) * um.two - 1);
                    val[j] = f[j] * n; vh[j] = fh[j] * n;
                }
            }
            int8_t *dst = (is_a ? na + (int64_t)row * ktot : nb + (int64_t)(row - cols_n) * ktot) + pp;
            *reinterpret_cast<uint32_t *>(dst) = pack4(val[0], val[1], val[2], val[3]);
            if (split) *reinterpret_cast<uint32_t *>(dst + kp) = pack4(vh[0], vh[1], vh[2], vh[3]);
        }
    }
}

int launch_update_operands(cudaStream_t st, int8_t *na, int8_t *nb, const int32_t *fit, int pairs, int kp, int rows_k,
                           int cols_n, int off_a, int off_b, int seed_base, uint32_t step_seed, int mask, int gaussian,
                           int split) {
    if (rows_k % UPD_ROWS_PER_BLOCK || cols_n % UPD_ROWS_PER_BLOCK) { set_error("update operand rows must come in groups of %d", UPD_ROWS_PER_BLOCK); return EGG_E_INVALID; }
    int gx = (kp / 4 + 255) / 256; if (gx > 32) gx = 32;
    dim3 grid((unsigned)gx, (unsigned)((rows_k + cols_n) / UPD_ROWS_PER_BLOCK));
    if (gaussian) update_operands_kernel<true><<<grid, 256, 0, st>>>(na, nb, fit, pairs, kp, rows_k, cols_n, off_a, off_b, seed_base, step_seed, mask, split, make_upd_mul());
    else update_operands_kernel<false><<<grid, 256, 0, st>>>(na, nb, fit, pairs, kp, rows_k, cols_n, off_a, off_b, seed_base, step_seed, mask, split, make_upd_mul());
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

int vote_gemm_splits(int rows_k, int cols_n, int kp, int num_sms) {
    const int bn = (rows_k % 256 == 0) ? 256 : 128;
    const int tiles = ((cols_n + GEMM_BM - 1) / GEMM_BM) * (rows_k / bn);
    const int num_kb = (kp + GEMM_BK - 1) / GEMM_BK;
    int want = (2 * num_sms + tiles - 1) / tiles;
    if (want > num_kb) want = num_kb;
    if (want > 64) want = 64;
    if (want < 1) want = 1;
    const int kb_per = (num_kb + want - 1) / want;
    return (num_kb + kb_per - 1) / kb_per;
}

// =========================================================================
// optimiser step from the vote matrices: one thread per packed word (4 weights of one output column)
// =========================================================================
__device__ __forceinline__ int4 sum_votes(const VoteApplyParams &p, int64_t word) {
    int4 v = *reinterpret_cast<const int4 *>(p.votes + word * 4);
    for (int s = 1; s < p.nsplits; s++) {
        const int4 u = *reinterpret_cast<const int4 *>(p.votes + (int64_t)s * p.split_stride + word * 4);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    return v;
}

__global__ void __launch_bounds__(256) adam_from_votes_kernel(const VoteApplyParams p) {
    const int64_t word = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t words = (int64_t)(p.rows_k >> 2) * p.cols_n;
    int changes = 0;
    if (word < words) {
        const int4 vt = sum_votes(p, word);
        const int vote[4] = {vt.x, vt.y, vt.z, vt.w};
        const int64_t idx = word * 4;
        const uint32_t wword = *reinterpret_cast<const uint32_t *>(p.w_packed + idx);
        float4 *st = reinterpret_cast<float4 *>(p.opt + idx * 3);
        const float4 s0 = st[0], s1 = st[1], s2 = st[2];
        float f[12] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w, s2.x, s2.y, s2.z, s2.w};
        uint32_t neww = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int w = (int)(int8_t)(wword >> (8 * j));
            const float g = -(float)vote[j];
            const int ch = adam_apply(f[3 * j], f[3 * j + 1], f[3 * j + 2], w, g, p.lr, p.beta1, p.beta2, p.eps, p.wd);
            changes += ch;
            neww |= (uint32_t)(w & 0xFF) << (8 * j);
        }
        *reinterpret_cast<uint32_t *>(p.w_packed + idx) = neww;
        st[0] = make_float4(f[0], f[1], f[2], f[3]);
        st[1] = make_float4(f[4], f[5], f[6], f[7]);
        st[2] = make_float4(f[8], f[9], f[10], f[11]);
    }
    changes = warp_sum(changes);
    if ((threadIdx.x & 31) == 0 && changes > 0) atomicAdd(p.total_updates, (unsigned long long)changes);
}

int launch_adam_from_votes(cudaStream_t st, const VoteApplyParams &p) {
    const int64_t words = (int64_t)(p.rows_k >> 2) * p.cols_n;
    adam_from_votes_kernel<<<(unsigned)((words + 255) / 256), 256, 0, st>>>(p);
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}
}  // namespace egg
