// Update reconstruction and optimiser step of a whole model (update_matrix/vector_adam_kernel, mgpu.cu:1040-1152): noise
// table, fitness masks, all vectors, then per batch of matrices the written operand, one vote GEMM and one optimiser pass.
#include "egg_update.cuh"
#include "egg_ptx.cuh"

#include <algorithm>
#include <map>
#include <cuda.h>
#include <limits.h>
#include <string.h>

namespace egg {

// ------------------------------------------------------------------ noise table
// Bound: the counter hash on the integer pipe, about 10^12 values a second; every distinct (seed, index) is hashed once,
// where a parameter-by-parameter update hashes one value per pair and operand row (40 times as many at H 256).
// The integer pipe is the busy one: additions are issued as multiply-adds, two of a hash's three shifts as the high word of a wide product
// (run-time multipliers keep them that), and signs are given to four values at once.  163 840 pairs at H 256: 125 -> 100 us (174 million values).
struct TabMul { int one; uint32_t up16, up19; };      // 1, 2^16, 2^19
__device__ __forceinline__ uint32_t mul_high(uint32_t x, uint32_t m) {
    uint64_t w;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(w) : "r"(x), "r"(m));
    return (uint32_t)(w >> 32);
}

template <bool GAUSS>
__global__ void __launch_bounds__(256) upd_table_kernel(int8_t *tab, int pitch, const int2 *chunks, int rows, int rows_per_block, uint32_t step_seed, int mask,
                                                        const TabMul um, unsigned long long *total, int *range, double *norm2, int nnorm) {
    chain_next();
    chain_wait();
    if (blockIdx.x == 0 && blockIdx.y == 0) {
        if (threadIdx.x == 0) { *total = 0; *range = 0; }
        for (int i = threadIdx.x; i < nnorm; i += blockDim.x) norm2[i] = 0.0;
    }
    const int2 ch = chunks[blockIdx.x];
    const int c = ch.x + (int)(threadIdx.x & 63) * 16;
    if ((int)(threadIdx.x & 63) * 16 >= ch.y) return;
    const int i1 = min(rows, (int)(blockIdx.y + 1) * rows_per_block);
    const uint32_t s0 = step_seed + (uint32_t)(c - UPD_ORIGIN);
    for (int i = (int)blockIdx.y * rows_per_block + (int)(threadIdx.x >> 6); i < i1; i += 4) {
        uint32_t w[4];
        const uint32_t base = s0 + (uint32_t)i * 0x9e3779b9u;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (GAUSS) {
                    v[k] = (uint32_t)noise_from_hash(s0 + (uint32_t)(4 * q + k), (uint32_t)i, mask, 1);
                } else {
                    uint32_t x = base * (uint32_t)um.one + (uint32_t)(4 * q + k);
                    x ^= x >> 16; x *= 0x85ebca6bu;
                    x ^= mul_high(x, um.up19); x *= 0xc2b2ae35u;
                    v[k] = x ^ mul_high(x, um.up16);
                }
            }
            uint32_t y = __byte_perm(__byte_perm(v[0], v[1], 0x0040), __byte_perm(v[2], v[3], 0x0040), 0x5410);
            if (!GAUSS) {
                // bytes: bit 0 the sign (set: positive), the mask's bits above it the magnitude, at most 127: 0x80 - m borrows from no neighbour
                uint32_t pos;
                asm("prmt.b32 %0, %1, 0, 0xba98;" : "=r"(pos) : "r"(y << 7));
                const uint32_t mag = (y >> 1) & ((uint32_t)mask * 0x01010101u);
                y = ((0x80808080u - (mag & ~pos)) ^ 0x80808080u) | (mag & pos);
            }
            w[q] = y;
        }
        *reinterpret_cast<uint4 *>(tab + (int64_t)i * pitch + c) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

int launch_upd_table(cudaStream_t st, const UpdPlan &pl, int8_t *tab, uint32_t step_seed, int mask, int gaussian, unsigned long long *total, int *range,
                     double *norm2) {
    // few columns (a small population): fewer rows per block so that the GPU fills
    int rpb = 64;
    while (rpb > 4 && (int64_t)pl.chunks.size() * (pl.W / rpb) < 1184) rpb >>= 1;
    const dim3 grid((unsigned)pl.chunks.size(), (unsigned)((pl.W + rpb - 1) / rpb));
    TabMul um; um.one = 1; um.up16 = 1u << 16; um.up19 = 1u << 19;
    if (gaussian) EGG_CUDA(launch_chained(upd_table_kernel<true>, grid, 256, 0, st, tab, pl.pitch, pl.d_chunks, pl.W, rpb, step_seed, mask, um, total, range, norm2, (int)pl.list.size()));
    else EGG_CUDA(launch_chained(upd_table_kernel<false>, grid, 256, 0, st, tab, pl.pitch, pl.d_chunks, pl.W, rpb, step_seed, mask, um, total, range, norm2, (int)pl.list.size()));
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// ------------------------------------------------------------------ fitness as byte masks, at every alignment, and as vector windows
__global__ void upd_masks_kernel(const int32_t *fit, int pairs, int kp, uint8_t *masks, int *range, int most, const UpdVec *vecs, int nvec, int vec_pad, int pitch,
                                 const UpdVecCols *vcols, int ncols, int8_t *vfit, int32_t *vvotes, int len_long) {
    chain_next();
    chain_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.y < 16) {
        const int j = t * 4;
        if (j >= kp) return;
        const int r = blockIdx.y;
        uint32_t pos = 0, neg = 0;
        int wide = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int p = j + k - r;
            const int f = (p >= 0 && p < pairs) ? fit[p] : 0;
            if (f > 0) pos |= 0xFFu << (8 * k);
            if (f < 0) neg |= 0xFFu << (8 * k);
            if (f > 1 || f < -1) wide |= (f > 127 || f < -127) ? 3 : 1;
            if (f > most || f < -most) wide |= 4;
        }
        *reinterpret_cast<uint32_t *>(masks + (int64_t)r * kp + j) = pos;
        *reinterpret_cast<uint32_t *>(masks + (int64_t)(16 + r) * kp + j) = neg;
        if (wide && r == 0) atomicOr(range, wide);
        return;
    }
    const int v = (int)blockIdx.y - 16;                  // one vector (or padding row): its fitness over every listed column
    for (int i = t; i < len_long; i += (int)(gridDim.x * blockDim.x)) vvotes[(int64_t)v * len_long + i] = 0;
    const int x = v < nvec ? vecs[v].x_a + vecs[v].r : 0;
    for (int e = t; e < ncols * 16; e += (int)(gridDim.x * blockDim.x)) {
        const int c = vcols[e >> 4].col + (e & 15) * 4;
        uint32_t w = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int p = c + k - x;
            const int f = (v < nvec && p >= 0 && p < pairs) ? fit[p] : 0;
            w |= (uint32_t)(f & 0xFF) << (8 * k);
        }
        *reinterpret_cast<uint32_t *>(vfit + (int64_t)v * pitch + c) = w;
    }
}

int64_t upd_vfit_bytes(const UpdPlan &pl) { return (int64_t)pl.vec_pad * pl.pitch; }
int64_t upd_vvotes_elems(const UpdPlan &pl) { return (int64_t)pl.vec_pad * pl.len_long; }

int launch_upd_masks(cudaStream_t st, const UpdPlan &pl, const int32_t *fit, uint8_t *masks, int8_t *vfit, int32_t *vvotes, int *range, int amp) {
    EGG_CUDA(launch_chained(upd_masks_kernel, dim3((unsigned)((pl.kp / 4 + 255) / 256), (unsigned)(16 + pl.vec_pad)), 256, 0, st, fit, pl.pairs, pl.kp, masks,
                            range, amp > 0 ? 127 / amp : INT_MAX, pl.d_vecs, (int)pl.vecs.size(), pl.vec_pad, pl.pitch, pl.d_vcols, (int)pl.vcols.size(), vfit, vvotes, pl.len_long));
    return EGG_OK;
}

// bytes of -n for four signed bytes (never -128)
__device__ __forceinline__ uint32_t neg4(uint32_t n) {
    const uint32_t m = ~n;
    return ((m & 0x7F7F7F7Fu) + 0x01010101u) ^ (m & 0x80808080u);
}
// fitness (as masks) times noise
__device__ __forceinline__ uint32_t fit_times(uint32_t n, uint32_t pos, uint32_t neg) { return (n & pos) | (neg4(n) & neg); }
// byte-wise product with general fitness values; beyond a byte it wraps
__device__ __forceinline__ uint32_t fit_times_wide(uint32_t n, const int32_t *fit, int p, int pairs) {
    uint32_t o = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int f = (p + k >= 0 && p + k < pairs) ? fit[p + k] : 0;
        o |= (uint32_t)((f * (int)(int8_t)(n >> (8 * k))) & 0xFF) << (8 * k);
    }
    return o;
}

// ------------------------------------------------------------------ vectors (update_vector_adam_kernel, mgpu.cu:1114-1152)
// vote_v[i] = Σ_p f_p noise(s_p + off_v, i) noise(s_p + off_v + 1, i): both factors are the same table row, one column apart, and
// the vectors differ only in where their window starts.  With g_i[c] = T[i][c] T[i][c + 1] all votes are one product
//     vote = g [rows x columns] * F [columns x vectors],  F[c][v] = f_(c - start of v)
// on the tensor cores; g is formed from the table words in registers, once for 32 vectors.  |g| <= 225 goes in as
// g = 2 (g >> 1) + (g & 1), two int8 operands.  Bound: forming g, about 5 instructions a table byte; 31 vectors over 163 840 pairs
// at H 256 take 75 us where a dot product per element and vector, bound by reading the table 24 times from L2, took 667.
constexpr int VC_TILES = 4;           // tiles of eight vectors per pass over the table

__device__ __forceinline__ void vc_mma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// products of 16 consecutive table bytes with their right neighbours: halves rounded down, and the low bits
__device__ __forceinline__ void vc_products(const int8_t *src, uint32_t (&half)[4], uint32_t (&low)[4]) {
    const uint4 a = *reinterpret_cast<const uint4 *>(src);
    const uint32_t w[5] = {a.x, a.y, a.z, a.w, *reinterpret_cast<const uint32_t *>(src + 16)};
    int s[17];
#pragma unroll
    for (int i = 0; i < 4; i++) { s[4 * i] = ptx::sx_byte0(w[i]); s[4 * i + 1] = ptx::sx_byte1(w[i]); s[4 * i + 2] = ptx::sx_byte2(w[i]); s[4 * i + 3] = (int)w[i] >> 24; }
    s[16] = ptx::sx_byte0(w[4]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        int p[4];
#pragma unroll
        for (int k = 0; k < 4; k++) p[k] = s[4 * i + k] * s[4 * i + k + 1];
        low[i] = __byte_perm(__byte_perm((uint32_t)p[0], (uint32_t)p[1], 0x0040), __byte_perm((uint32_t)p[2], (uint32_t)p[3], 0x0040), 0x5410) & 0x01010101u;
        half[i] = __byte_perm(__byte_perm((uint32_t)(p[0] >> 1), (uint32_t)(p[1] >> 1), 0x0040), __byte_perm((uint32_t)(p[2] >> 1), (uint32_t)(p[3] >> 1), 0x0040), 0x5410);
    }
}

// block: 16 table rows, every gridDim.x-th group of eight listed column blocks (one per warp), VC_TILES tiles of vectors
__global__ void __launch_bounds__(256) upd_vec_votes_kernel(const int8_t *tab, int pitch, const int8_t *vfit, const UpdVecCols *cols, int ncols, int vec_pad,
                                                            int vec_long, int len_short, int len_long, int32_t *votes, const int *range) {
    chain_next();
    chain_wait();
    if (*range & 2) return;                              // the optimiser kernel sums these itself
    __shared__ int red[8][VC_TILES * 4][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int row0 = (int)blockIdx.y * 16, tile0 = (int)blockIdx.z * VC_TILES;
    const int tiles_all = (row0 < len_short ? vec_pad : vec_long + 7) / 8;       // rows beyond the short vectors: the long ones only
    const int nt = min(VC_TILES, tiles_all - tile0);
    if (nt <= 0) return;
    const uint32_t want = (1u << nt) - 1;
    int ah[VC_TILES][4] = {}, al[VC_TILES][4] = {};
    const int8_t *r0 = tab + (int64_t)(row0 + g) * pitch + 16 * q, *r1 = r0 + (int64_t)8 * pitch;
    const int8_t *fb = vfit + (int64_t)(tile0 * 8 + g) * pitch + 16 * q;
    for (int e = (int)blockIdx.x * 8 + warp; e < ncols; e += (int)gridDim.x * 8) {
        const UpdVecCols vc = cols[e];
        const uint32_t on = (vc.tiles[tile0 >> 5] >> (tile0 & 31)) & want;
        if (!on) continue;
        uint32_t h0[4], l0[4], h1[4], l1[4];
        uint4 b[VC_TILES];
#pragma unroll
        for (int t = 0; t < VC_TILES; t++) {
            b[t] = make_uint4(0, 0, 0, 0);
            if (on >> t & 1) b[t] = *reinterpret_cast<const uint4 *>(fb + (int64_t)t * 8 * pitch + vc.col);
        }
        vc_products(r0 + vc.col, h0, l0);
        vc_products(r1 + vc.col, h1, l1);
#pragma unroll
        for (int t = 0; t < VC_TILES; t++) {
            if (!(on >> t & 1)) continue;
            vc_mma(ah[t], h0[0], h1[0], h0[1], h1[1], b[t].x, b[t].y);
            vc_mma(al[t], l0[0], l1[0], l0[1], l1[1], b[t].x, b[t].y);
            vc_mma(ah[t], h0[2], h1[2], h0[3], h1[3], b[t].z, b[t].w);
            vc_mma(al[t], l0[2], l1[2], l0[3], l1[3], b[t].z, b[t].w);
        }
    }
#pragma unroll
    for (int t = 0; t < VC_TILES; t++)
#pragma unroll
        for (int i = 0; i < 4; i++) red[warp][t * 4 + i][lane] = 2 * ah[t][i] + al[t][i];
    __syncthreads();
    for (int j = threadIdx.x; j < nt * 4 * 32; j += 256) {
        const int ti = j >> 5, l = j & 31;
        int sum = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) sum += red[w][ti][l];
        const int v = (tile0 + (ti >> 2)) * 8 + 2 * (l & 3) + (ti & 1), row = row0 + (l >> 2) + 8 * ((ti >> 1) & 1);
        if (sum) atomicAdd(&votes[(int64_t)v * len_long + row], sum);
    }
}

// The optimiser step: four consecutive elements of one vector per warp, votes as summed above.  Where they were not (Gaussian noise,
// fitness beyond int8) the warp sums them over the pairs itself; groups are
// ordered by index first, because all vectors share row i of the table.
constexpr int VEC_GROUP = 4;

__global__ void __launch_bounds__(256) upd_vectors_kernel(const UpdVec *vecs, int nvec, int vec_long, int len_short, int groups, const int8_t *tab, int pitch,
                                                          const uint8_t *masks, int kp, const int *range, const int32_t *vvotes, int len_long, const int32_t *fit, int pairs,
                                                          int8_t *model, uint8_t *opt, const UpdHyper h, unsigned long long *total, uint8_t *changed) {
    chain_next();
    chain_wait();
    const int gidx = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (gidx >= groups) return;
    const int both = nvec * (len_short / VEC_GROUP);         // groups whose index every vector has
    int vi, i0;
    if (gidx < both) { i0 = gidx / nvec * VEC_GROUP; vi = gidx % nvec; }
    else { i0 = len_short + (gidx - both) / vec_long * VEC_GROUP; vi = (gidx - both) % vec_long; }
    const UpdVec v = vecs[vi];
    const int rg = *range;
    const bool wide = rg != 0, summed = vvotes && !(rg & 2);
    int acc[VEC_GROUP] = {};
    const uint8_t *mp = masks + (int64_t)v.r * kp, *mn = masks + (int64_t)(16 + v.r) * kp;
    const int8_t *row = tab + (int64_t)i0 * pitch + v.x_a;
    for (int j = lane * 16; j < kp && !summed && !wide; j += 512) {
        const uint4 ps = *reinterpret_cast<const uint4 *>(mp + j), ng = *reinterpret_cast<const uint4 *>(mn + j);
#pragma unroll
        for (int e = 0; e < VEC_GROUP; e++) {
            const int8_t *src = row + (int64_t)e * pitch + j;
            const uint4 a = *reinterpret_cast<const uint4 *>(src);
            const uint32_t a4 = *reinterpret_cast<const uint32_t *>(src + 16);
            const uint32_t b0 = __funnelshift_r(a.x, a.y, 8), b1 = __funnelshift_r(a.y, a.z, 8), b2 = __funnelshift_r(a.z, a.w, 8), b3 = __funnelshift_r(a.w, a4, 8);
            acc[e] = __dp4a((int)fit_times(a.x, ps.x, ng.x), (int)b0, acc[e]);
            acc[e] = __dp4a((int)fit_times(a.y, ps.y, ng.y), (int)b1, acc[e]);
            acc[e] = __dp4a((int)fit_times(a.z, ps.z, ng.z), (int)b2, acc[e]);
            acc[e] = __dp4a((int)fit_times(a.w, ps.w, ng.w), (int)b3, acc[e]);
        }
    }
    // general fitness: four pairs at a time, their fitness loaded once for the group's elements; consecutive lanes take consecutive
    // words (an update with fitness to 200 at H 1024, 131 072 pairs: 10.6 ms with 16 pairs and a load per element, 7.5 so)
    for (int j = lane * 4; j < kp && !summed && wide; j += 128) {
        int f[4];
#pragma unroll
        for (int k = 0; k < 4; k++) { const int p = j + k - v.r; f[k] = p >= 0 && p < pairs ? fit[p] : 0; }
#pragma unroll
        for (int e = 0; e < VEC_GROUP; e++) {
            const int8_t *src = row + (int64_t)e * pitch + j;
            const uint32_t a = *reinterpret_cast<const uint32_t *>(src), b = __funnelshift_r(a, *reinterpret_cast<const uint32_t *>(src + 4), 8);
            acc[e] += f[0] * (ptx::sx_byte0(a) * ptx::sx_byte0(b)) + f[1] * (ptx::sx_byte1(a) * ptx::sx_byte1(b)) + f[2] * (ptx::sx_byte2(a) * ptx::sx_byte2(b)) +
                      f[3] * (((int)a >> 24) * ((int)b >> 24));
        }
    }
#pragma unroll
    for (int e = 0; e < VEC_GROUP; e++) acc[e] = __reduce_add_sync(0xFFFFFFFFu, acc[e]);
    int ch = 0;
    if (lane < VEC_GROUP) {
        int vote = 0;
#pragma unroll
        for (int e = 0; e < VEC_GROUP; e++) if (lane == e) vote = acc[e];
        const int i = i0 + lane;
        if (summed) vote = vvotes[(int64_t)vi * len_long + i];
        float *o = reinterpret_cast<float *>(opt + v.opt_off) + 3 * (int64_t)i;
        float m = o[0], s = o[1], a = o[2];
        int w = model[v.model_off + i];
        ch = adam_apply(m, s, a, w, -(float)vote, h.lr * v.lr_scale, h.beta1, h.beta2, h.eps, h.wd);
        o[0] = m; o[1] = s; o[2] = a;
        model[v.model_off + i] = (int8_t)w;
        if (ch && changed) changed[v.ov + i] = 1;
    }
    ch = __reduce_add_sync(0xFFFFFFFFu, ch);
    if (lane == 0 && ch) atomicAdd(total, (unsigned long long)ch);
}

int launch_upd_vectors(cudaStream_t st, const UpdPlan &pl, const int8_t *tab, const uint8_t *masks, const int8_t *vfit, int32_t *vvotes, const int *range,
                       const int32_t *fit, int gaussian, int8_t *model, uint8_t *opt, const UpdHyper &h, unsigned long long *total, uint8_t *changed, int num_sms) {
    const int nvec = (int)pl.vecs.size();
    if (!nvec) return EGG_OK;
    const bool product = !gaussian;
    if (product) {
        const int rows = pl.len_long / 16, z = (pl.vec_pad / 8 + VC_TILES - 1) / VC_TILES, ncols = (int)pl.vcols.size();
        int gx = (num_sms * 6 + rows * z - 1) / (rows * z);
        if (gx > (ncols + 7) / 8) gx = (ncols + 7) / 8;
        EGG_CUDA(launch_chained(upd_vec_votes_kernel, dim3((unsigned)gx, (unsigned)rows, (unsigned)z), 256, 0, st, tab, pl.pitch, vfit, pl.d_vcols, ncols, pl.vec_pad,
                                pl.len_long == pl.len_short ? 0 : pl.vec_long, pl.len_short, pl.len_long, vvotes, range));
    }
    const int groups = nvec * (pl.len_short / VEC_GROUP) + pl.vec_long * ((pl.len_long - pl.len_short) / VEC_GROUP);
    EGG_CUDA(launch_chained(upd_vectors_kernel, (groups + 7) / 8, 256, 0, st, pl.d_vecs, nvec, pl.vec_long, pl.len_short, groups, tab, pl.pitch, masks, pl.kp, range,
                            product ? vvotes : nullptr, pl.len_long, fit, pl.pairs, model, opt, h, total, changed));
    return EGG_OK;
}

// ------------------------------------------------------------------ the written operand: fitness times noise
// FN[row][j] = f[j - r] * T[i][x_fn + j]; 16 bytes per thread and row.  Bound: memory, one byte read and written per pair and row;
// it takes many warps to get near (163 840 pairs at H 256: 463 us with 3 blocks per SM, 327 with 5, 280 with 6 and two rows at a
// time; 8 blocks spill).  Consecutive blocks take the rows of one stretch of pairs, so that the table is read once.
constexpr int FN_ROWS = 8;            // rows per block: the masks are read once for all of them

__global__ void __launch_bounds__(256, 6) upd_operands_kernel(const UpdMat *mats, int nmats, const int8_t *tab, int pitch, const uint8_t *masks, int kp,
                                                           const int *range, const int32_t *fit, int pairs, int rows1, int8_t *fn) {
    chain_next();
    int row0 = (int)blockIdx.x * FN_ROWS;
    auto find = [&](int form) {
        int lo = 0, hi = nmats - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (mats[mid].form[form].fn_row0 <= row0) lo = mid; else hi = mid - 1;
        }
        return mats[lo].form[form];
    };
    UpdForm m = find(0);                          // (descriptors are older than the chain)
    chain_wait();
    const int rg = *range;
    const bool wide = rg != 0;
    // the grid covers form 0's rows; products that wrap take form 1's, more of them, in as many trips as it needs
    const int rows = rg & 4 ? rows1 : row0 + 1;
    for (; row0 < rows; row0 += (int)gridDim.x * FN_ROWS) {
        if (rg & 4) m = find(1);
        const int x = m.x_fn, sh = (x & 3) * 8, r = m.r;
        const bool by2 = x & 8, by1 = x & 4;
        const int8_t *src0 = tab + (int64_t)(row0 - m.fn_row0) * pitch + (x & ~15);
        const uint8_t *mp = masks + (int64_t)r * kp, *mn = masks + (int64_t)(16 + r) * kp;
        for (int j = (int)(blockIdx.y * blockDim.x + threadIdx.x) * 16; j < kp; j += (int)(gridDim.y * blockDim.x) * 16) {
            const uint4 ps = *reinterpret_cast<const uint4 *>(mp + j), ng = *reinterpret_cast<const uint4 *>(mn + j);
#pragma unroll 2
            for (int e = 0; e < FN_ROWS; e++) {
                // 16 bytes from any byte offset: two aligned words of 16, shifted by words, then by bytes
                const uint4 *src = reinterpret_cast<const uint4 *>(src0 + (int64_t)e * pitch + j);
                const uint4 a = src[0], b = src[1];
                uint32_t w0 = a.x, w1 = a.y, w2 = a.z, w3 = a.w, w4 = b.x, w5 = b.y;
                if (by2) { w0 = w2; w1 = w3; w2 = w4; w3 = w5; w4 = b.z; w5 = b.w; }
                if (by1) { w0 = w1; w1 = w2; w2 = w3; w3 = w4; w4 = w5; }
                uint4 n = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
                if (!wide) n = make_uint4(fit_times(n.x, ps.x, ng.x), fit_times(n.y, ps.y, ng.y), fit_times(n.z, ps.z, ng.z), fit_times(n.w, ps.w, ng.w));
                else n = make_uint4(fit_times_wide(n.x, fit, j - r, pairs), fit_times_wide(n.y, fit, j - r + 4, pairs), fit_times_wide(n.z, fit, j - r + 8, pairs),
                                    fit_times_wide(n.w, fit, j - r + 12, pairs));
                *reinterpret_cast<uint4 *>(fn + (int64_t)(row0 + e) * kp + j) = n;
            }
        }
    }
}

int launch_upd_operands(cudaStream_t st, const UpdPlan &pl, const UpdBatch &b, const int8_t *tab, const uint8_t *masks, const int *range,
                        const int32_t *fit, int8_t *fn) {
    int gy = (pl.kp / 16 + 255) / 256;
    if (gy > 65535) gy = 65535;
    EGG_CUDA(launch_chained(upd_operands_kernel, dim3((unsigned)(b.fn_rows[0] / FN_ROWS), (unsigned)gy), 256, 0, st, pl.d_mats + b.first, b.count, tab, pl.pitch, masks, pl.kp, range,
                            fit, pl.pairs, b.fn_rows[1], fn));
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// ------------------------------------------------------------------ vote GEMM over a batch of matrices
// votes_m[k][n] = Σ_j A_m[n][j] B_m[k][j], one operand read from the table in place.  Persistent; work item = (split of the
// contraction, 128 x 256 tile of some matrix); TMA -> 4-stage ring -> tcgen05 kind::i8 -> two TMEM accumulator stages -> eight
// epilogue warps that store int32 votes in the packed weight order.  One launch for all matrices of a batch: a model of 27
// matrices is 114 to 456 tiles, where each matrix alone left the GPU mostly idle or cut its contraction into 8 to 64 pieces.
// A tile's last 128 columns may lie beyond its matrix (rows_k an odd multiple of 128): they multiply whatever rows follow and
// are not stored.
// CG == 2: pairs of blocks form 256 x 256 tiles together (cta_group::2), each block with 128 rows of both operands; the second half of a
// matrix's last tile may lie beyond it in the same way.
constexpr int UV_BM = 128, UV_BN = 256, UV_BK = 128, UV_EPI_WARPS = 8;
constexpr int UV_THREADS = 64 + UV_EPI_WARPS * 32;
constexpr int UV_MAX_MATS = 512;

template <int CG>
struct UpdVoteSmem {
    static constexpr int ST = CG == 2 ? 6 : 4;          // ring stages
    alignas(1024) uint8_t a[ST][UV_BM * UV_BK];
    alignas(1024) uint8_t b[ST][UV_BN / CG * UV_BK];
    alignas(8) uint64_t full[ST], empty[ST], tmem_full[2], tmem_empty[2];
    int tile0[UV_MAX_MATS];
    uint32_t tmem_base;
    volatile int abort_flag;
};

struct UpdVoteParams {
    const UpdMat *mats; int nmats, tiles, splits, num_kb;
    const int *range;
    int32_t *votes; int64_t split_stride;
    int *err;
};

template <int CG>
__global__ void __launch_bounds__(UV_THREADS, 1)
upd_votes_kernel(const __grid_constant__ CUtensorMap tab_a, const __grid_constant__ CUtensorMap tab_b, const __grid_constant__ CUtensorMap fn_a,
                 const __grid_constant__ CUtensorMap fn_b, const UpdVoteParams p) {
    extern __shared__ uint8_t uv_raw[];
    using Smem = UpdVoteSmem<CG>;
    constexpr int ST = Smem::ST;
    Smem &sm = *reinterpret_cast<Smem *>((reinterpret_cast<uintptr_t>(uv_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    chain_next();
    const int items = p.tiles * p.splits, kb_per = (p.num_kb + p.splits - 1) / p.splits;
    const int prow = CG == 2 ? (int)(blockIdx.x & 1) : 0;           // this block of the pair (clusters are consecutive blocks)
    const int first_item = (int)blockIdx.x / CG, item_step = (int)gridDim.x / CG;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) { ptx::mbar_init(&sm.full[s], 1); ptx::mbar_init(&sm.empty[s], 1); }
        for (int a = 0; a < 2; a++) { ptx::mbar_init(&sm.tmem_full[a], 1); ptx::mbar_init(&sm.tmem_empty[a], CG * UV_EPI_WARPS); }
        sm.abort_flag = 0;
        ptx::fence_barrier_init();
    }
    for (int i = threadIdx.x; i < p.nmats; i += UV_THREADS) sm.tile0[i] = p.mats[i].tile0;
    if (warp == 1) {
        if (CG == 2) ptx::tmem_alloc_pair(&sm.tmem_base, 512);
        else {
            ptx::tmem_alloc(&sm.tmem_base, 512);
            ptx::tmem_relinquish();
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    if (CG == 2) ptx::cluster_sync_all();          // the other block's barriers exist before anything arrives on them
    chain_wait();
    const uint32_t tmem_base = sm.tmem_base;
    auto find = [&](int tile) {                   // matrix that owns the tile
        int lo = 0, hi = p.nmats - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sm.tile0[mid] <= tile) lo = mid; else hi = mid - 1;
        }
        return lo;
    };
    auto fail = [&](int code) {
        sm.abort_flag = 1;
        if (p.err) atomicCAS(p.err, 0, code);
    };
    if (warp == 0) {
        if (ptx::elect_one()) {
            uint32_t it = 0;
            bool ok = true;
            const int form = *p.range >> 2 & 1;
            const uint32_t full_s = CG == 2 ? ptx::mapa_u32(ptx::smem_u32(sm.full), 0u) : 0u;          // of the even block
            for (int item = first_item; item < items && ok; item += item_step) {
                const int split = item / p.tiles, tile = item - split * p.tiles;
                const UpdMat &m = p.mats[find(tile)];
                const UpdForm f = m.form[form];
                const int local = tile - m.tile0, tm = local / m.tiles_n, tn = local - tm * m.tiles_n;
                const int ya = (tm * CG + prow) * UV_BM + (f.fn_is_n ? f.fn_row0 : 0), yb = tn * UV_BN + prow * (UV_BN / CG) + (f.fn_is_n ? 0 : f.fn_row0);
                const int xa = f.fn_is_n ? 0 : f.x_tab, xb = f.fn_is_n ? f.x_tab : 0;
                const CUtensorMap *ta = f.fn_is_n ? &fn_a : &tab_a, *tb = f.fn_is_n ? &tab_b : &fn_b;
                const int kb1 = min(p.num_kb, (split + 1) * kb_per);
                for (int kb = split * kb_per; kb < kb1; kb++, it++) {
                    const int s = it % ST;
                    if (!ptx::mbar_wait(&sm.empty[s], ((it / ST) & 1) ^ 1) || sm.abort_flag) { fail(DEV_TIMEOUT_EMPTY); ok = false; break; }
                    if (CG == 2) {
                        if (prow == 0) ptx::mbar_arrive_expect_tx(&sm.full[s], 2 * (UV_BM + UV_BN / CG) * UV_BK);          // both blocks' bytes
                        ptx::tma_load_2d_pair(sm.a[s], ta, full_s + 8 * s, xa + kb * UV_BK, ya);
                        ptx::tma_load_2d_pair(sm.b[s], tb, full_s + 8 * s, xb + kb * UV_BK, yb);
                    } else {
                        ptx::mbar_arrive_expect_tx(&sm.full[s], (UV_BM + UV_BN) * UV_BK);
                        ptx::tma_load_2d(sm.a[s], ta, &sm.full[s], xa + kb * UV_BK, ya);
                        ptx::tma_load_2d(sm.b[s], tb, &sm.full[s], xb + kb * UV_BK, yb);
                    }
                }
            }
            if (!ok) {   // let copies already in flight land before the block tears down
                const uint64_t t0 = ptx::globaltimer();
                while (ptx::globaltimer() - t0 < 200000ull) __nanosleep(1000);
            }
        }
    } else if (warp == 1) {
        if (prow == 0 && ptx::elect_one()) {
            constexpr uint32_t idesc = ptx::make_idesc_i8(CG * UV_BM, UV_BN);
            uint32_t it = 0, tc = 0;
            bool ok = true;
            for (int item = first_item; item < items && ok; item += item_step, tc++) {
                const int split = item / p.tiles, as = tc & 1;
                if (!ptx::mbar_wait(&sm.tmem_empty[as], ((tc >> 1) & 1) ^ 1) || sm.abort_flag) { fail(DEV_TIMEOUT_TMEM_EMPTY); break; }
                ptx::tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(as * UV_BN);
                const int kb0 = split * kb_per, kb1 = min(p.num_kb, kb0 + kb_per);
                for (int kb = kb0; kb < kb1; kb++, it++) {
                    const int s = it % ST;
                    if (!ptx::mbar_wait(&sm.full[s], (it / ST) & 1) || sm.abort_flag) { fail(DEV_TIMEOUT_FULL); ok = false; break; }
                    ptx::tc_fence_after();
                    const uint64_t da = ptx::make_smem_desc_sw128(ptx::smem_u32(sm.a[s])), db = ptx::make_smem_desc_sw128(ptx::smem_u32(sm.b[s]));
#pragma unroll
                    for (int k = 0; k < UV_BK / 32; k++) {
                        if (CG == 2) ptx::mma_i8_pair(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
                        else ptx::mma_i8(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
                    }
                    if (CG == 2) ptx::mma_commit_pair(&sm.empty[s], 0); else ptx::mma_commit(&sm.empty[s]);
                }
                if (ok) {
                    if (CG == 2) ptx::mma_commit_pair(&sm.tmem_full[as], 0); else ptx::mma_commit(&sm.tmem_full[as]);
                }
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;         // TMEM lane quarter, half of the tile's columns
        const uint32_t tmem_empty_s = CG == 2 ? ptx::mapa_u32(ptx::smem_u32(sm.tmem_empty), 0u) : 0u;          // of the even block
        uint32_t tc = 0;
        for (int item = first_item; item < items; item += item_step, tc++) {
            const int split = item / p.tiles, tile = item - split * p.tiles, as = tc & 1;
            const UpdMat &m = p.mats[find(tile)];
            const int local = tile - m.tile0, tm = local / m.tiles_n, tn = local - tm * m.tiles_n;
            const int n = (tm * CG + prow) * UV_BM + quarter * 32 + lane, kbase = tn * UV_BN + half * 128;
            const int cols_n = m.cols_n, rows_k = m.rows_k;
            int32_t *vout = p.votes + (int64_t)split * p.split_stride + m.votes_off;
            const bool ok = ptx::mbar_wait(&sm.tmem_full[as], (tc >> 1) & 1) && !sm.abort_flag;
            if (!__all_sync(0xFFFFFFFFu, ok)) { if (lane == 0) fail(DEV_TIMEOUT_TMEM_FULL); break; }
            ptx::tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(as * UV_BN + half * 128);
#pragma unroll 1
            for (int c = 0; c < 128 && kbase + c < rows_k && (CG == 1 || n < cols_n); c += 32) {
                uint32_t v[32];
                ptx::tmem_ld32(taddr + c, v);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int64_t word = (int64_t)(((kbase + c) >> 2) + q) * cols_n + n;
                    *reinterpret_cast<int4 *>(vout + word * 4) = make_int4((int)v[4 * q], (int)v[4 * q + 1], (int)v[4 * q + 2], (int)v[4 * q + 3]);
                }
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (CG == 2) ptx::mbar_arrive_peer(tmem_empty_s + 8 * as); else ptx::mbar_arrive(&sm.tmem_empty[as]);
            }
        }
    }
    __syncwarp();
    ptx::tc_fence_before();
    __syncthreads();
    if (CG == 2) ptx::cluster_sync_all();          // a pair gives its tensor memory back together, after both blocks' reads
    if (warp == 1) {
        ptx::tc_fence_after();
        if (CG == 2) ptx::tmem_dealloc_pair(tmem_base, 512); else ptx::tmem_dealloc(tmem_base, 512);
    }
    if (CG == 2) { __syncwarp(); ptx::cluster_sync_all(); }          // neither block retires before the other is done with its memory
}

int upd_init() {
    static bool done[EGG_MAX_DEVICES] = {};
    bool &d = done[current_device_slot()];
    if (d) return EGG_OK;
    EGG_CUDA(cudaFuncSetAttribute(upd_votes_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(UpdVoteSmem<1>) + 1024));
    EGG_CUDA(cudaFuncSetAttribute(upd_votes_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(UpdVoteSmem<2>) + 1024));
    d = true;
    return EGG_OK;
}

int launch_upd_votes(cudaStream_t st, const UpdPlan &pl, const UpdBatch &b, const int8_t *tab, const int8_t *fn, const int *range, int32_t *votes, int *err, int num_sms) {
    CUtensorMap ta, tb, fa, fb;
    int rc;
    const uint64_t fn_rows = (uint64_t)std::max(b.fn_rows[0], b.fn_rows[1]);
    const uint32_t b_rows = UV_BN / pl.cg;
    if ((rc = upd_tensor_map(&ta, tab, (uint64_t)pl.W, (uint64_t)pl.pitch, UV_BM)) || (rc = upd_tensor_map(&tb, tab, (uint64_t)pl.W, (uint64_t)pl.pitch, b_rows)) ||
        (rc = upd_tensor_map(&fa, fn, fn_rows, (uint64_t)pl.kp, UV_BM)) || (rc = upd_tensor_map(&fb, fn, fn_rows, (uint64_t)pl.kp, b_rows)))
        return rc;
    UpdVoteParams p;
    p.mats = pl.d_mats + b.first; p.nmats = b.count; p.tiles = b.tiles; p.splits = b.splits; p.num_kb = pl.kp / UV_BK;
    p.range = range; p.votes = votes; p.split_stride = b.votes; p.err = err;
    const int items = b.tiles * b.splits;
    if (pl.cg == 1) {
        EGG_CUDA(launch_chained(upd_votes_kernel<1>, items < num_sms ? items : num_sms, UV_THREADS, sizeof(UpdVoteSmem<1>) + 1024, st, ta, tb, fa, fb, p));
    } else {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        cfg.blockDim = dim3(UV_THREADS); cfg.dynamicSmemBytes = sizeof(UpdVoteSmem<2>) + 1024; cfg.stream = st;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr; cfg.numAttrs = t_chain ? 2 : 1;
        const int most = num_sms / 2;             // where fewer pairs are resident, the others follow
        cfg.gridDim = dim3((unsigned)(2 * (items < most ? items : most)));
        EGG_CUDA(cudaLaunchKernelEx(&cfg, upd_votes_kernel<2>, ta, tb, fa, fb, p));
    }
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// ------------------------------------------------------------------ ES-AdamW of a batch (mgpu.cu:1040-1064, 1100-1110)
// A block owns 32 outputs x 128 inputs: votes, weights and state stream through once, and the new weights also leave in the
// K-major copy the evaluation reads (through shared memory, whole 128-byte rows), which used to be a pass of its own.
// Bound: memory, 27 bytes per weight and 4 per partial vote.
__global__ void __launch_bounds__(256) upd_adam_kernel(const UpdMat *mats, int nmats, const int32_t *votes, int splits, int64_t split_stride, int8_t *model,
                                                       uint8_t *opt, int8_t *shadow, const UpdHyper h, unsigned long long *total, uint8_t *changed) {
    chain_next();
    __shared__ uint32_t tile[32][33];
    __shared__ int s_changes;
    int lo = 0, hi = nmats - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (mats[mid].blk0 <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    const UpdMat m = mats[lo];                    // (descriptors are older than the chain)
    chain_wait();
    if (m.muon) return;
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int local = (int)blockIdx.x - m.blk0, bn = m.cols_n / 32, n = (local % bn) * 32 + lane, kq0 = (local / bn) * 32;
    const float lr = h.lr * m.lr_scale;
    if (threadIdx.x == 0) s_changes = 0;
    __syncthreads();
    int changes = 0;
    bool ch_n = false;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int kq = kq0 + ty + 8 * i;
        const int64_t word = (int64_t)kq * m.cols_n + n;
        int4 vt = *reinterpret_cast<const int4 *>(votes + m.votes_off + word * 4);
        for (int s = 1; s < splits; s++) {
            const int4 u = *reinterpret_cast<const int4 *>(votes + (int64_t)s * split_stride + m.votes_off + word * 4);
            vt.x += u.x; vt.y += u.y; vt.z += u.z; vt.w += u.w;
        }
        const int vote[4] = {vt.x, vt.y, vt.z, vt.w};
        uint32_t *wp = reinterpret_cast<uint32_t *>(model + m.model_off) + word;
        float4 *sp = reinterpret_cast<float4 *>(opt + m.opt_off) + word * 3;
        const uint32_t wword = *wp;
        const float4 s0 = sp[0], s1 = sp[1], s2 = sp[2];
        float f[12] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w, s2.x, s2.y, s2.z, s2.w};
        uint32_t neww = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int w = (int)(int8_t)(wword >> (8 * j));
            const int ch = adam_apply(f[3 * j], f[3 * j + 1], f[3 * j + 2], w, -(float)vote[j], lr, h.beta1, h.beta2, h.eps, h.wd);
            changes += ch;
            if (ch && changed) { changed[m.ov_in + 4 * kq + j] = 1; ch_n = true; }        // adam.cuh:77-83
            neww |= (uint32_t)(w & 0xFF) << (8 * j);
        }
        *wp = neww;
        sp[0] = make_float4(f[0], f[1], f[2], f[3]);
        sp[1] = make_float4(f[4], f[5], f[6], f[7]);
        sp[2] = make_float4(f[8], f[9], f[10], f[11]);
        tile[ty + 8 * i][lane] = neww;
    }
    if (ch_n) changed[m.ov_out + n] = 1;
    changes = __reduce_add_sync(0xFFFFFFFFu, changes);
    if (lane == 0 && changes) atomicAdd(&s_changes, changes);
    __syncthreads();
    int8_t *sh = shadow + m.shadow_off;
    const int n0 = n - lane;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int nn = ty + 8 * i;
        *reinterpret_cast<uint32_t *>(sh + (int64_t)(n0 + nn) * m.rows_k + 4 * (kq0 + lane)) = tile[lane][nn];
    }
    if (threadIdx.x == 0 && s_changes) atomicAdd(total, (unsigned long long)s_changes);
}

int launch_upd_adam(cudaStream_t st, const UpdPlan &pl, const UpdBatch &b, const int32_t *votes, int8_t *model, uint8_t *opt, int8_t *shadow,
                    const UpdHyper &h, unsigned long long *total, uint8_t *changed) {
    EGG_CUDA(launch_chained(upd_adam_kernel, (unsigned)b.blocks, 256, 0, st, pl.d_mats + b.first, b.count, votes, b.splits, b.votes, model, opt, shadow, h, total, changed));
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

__global__ void overlay_step_all_kernel(int8_t *ov, uint8_t *changed, const uint8_t *active, int n, int inc, int dec) {
    chain_next();
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !active[i]) return;
    int v = ov[i];
    if (changed[i]) { v += inc; if (v > 127) v = 127; } else { v -= dec; if (v < -127) v = -127; }
    ov[i] = (int8_t)v;
    changed[i] = 0;
}
int launch_overlay_step_all(cudaStream_t st, int8_t *ov, uint8_t *changed, const uint8_t *active, int n, int inc, int dec) {
    EGG_CUDA(launch_chained(overlay_step_all_kernel, (n + 255) / 256, 256, 0, st, ov, changed, active, n, inc, dec));
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// ------------------------------------------------------------------ plan
// Workspace of one batch: enough for every model of up to a few dozen million weights at once; larger ones take turns.
constexpr int64_t UPD_FN_BYTES = 1ll << 30, UPD_VOTE_ELEMS = 128ll << 20;

int64_t upd_table_bytes(const UpdPlan &pl) { return (int64_t)pl.W * pl.pitch + 64; }
int64_t upd_mask_bytes(const UpdPlan &pl) { return 32ll * pl.kp; }

int upd_plan_upload(UpdPlan &pl, uint8_t *dev, cudaStream_t st) {
    EGG_CUDA(cudaMemcpyAsync(dev, pl.descriptors.data(), pl.descriptors.size(), cudaMemcpyHostToDevice, st));
    pl.d_mats = reinterpret_cast<UpdMat *>(dev);
    pl.d_vecs = reinterpret_cast<UpdVec *>(dev + pl.o_vecs);
    pl.d_chunks = reinterpret_cast<int2 *>(dev + pl.o_chunks);
    pl.d_list = reinterpret_cast<int *>(dev + pl.o_list);
    pl.d_vcols = reinterpret_cast<UpdVecCols *>(dev + pl.o_vcols);
    return EGG_OK;
}

int upd_plan_build(UpdPlan &pl, const std::vector<ParamDesc> &params, const std::vector<char> &use, int hidden, int vocab, int pairs, int num_sms) {
    pl = UpdPlan();
    pl.pairs = pairs;
    pl.kp = (pairs + 15 + 127) / 128 * 128;
    pl.W = std::max(4 * hidden, vocab);
    // Vote tiles in pairs of blocks: half of one operand's traffic from L2, which bounds the product.  Per tile of 128 columns they take 0.73
    // to 0.82 of the time (163 840 pairs, H 256: 581 -> 427 us; 131 072, H 1024: 12.2 -> 10.0 ms; 20 480, H 512: 292 -> 211 us; 4096, H 256: 23 -> 19),
    // so that a model takes them unless odd multiples of 128 outputs leave more than a fifth of their halves empty, and not for few pairs, which a
    // launch of clusters does not pay for: whole updates of 32 to 368 pairs 1 to 3 us longer at H 256 to 1024 (H 256, 2 layers: 46.1 -> 47.2; H 896
    // 228.5 -> 231.5; at most 1.4 shorter at H 512, 4 layers), of 480 (four blocks of the contraction) 1.5 shorter at H 512, 2.8 at 1024, of 512 up to 20.
    int64_t single = 0, paired = 0;
    for (const ParamDesc &d : params)
        if (d.rows_k) {
            const int64_t tn = (d.rows_k + UV_BN - 1) / UV_BN;
            single += d.cols_n / UV_BM * tn; paired += (d.cols_n + 2 * UV_BM - 1) / (2 * UV_BM) * 2 * tn;
        }
    pl.cg = pl.kp >= 512 && 5 * single >= 4 * paired ? 2 : 1;
    std::vector<std::pair<int, int>> need;                   // table columns [first, last)
    auto want = [&](int s) { need.push_back({s & ~127, (s + UPD_ORIGIN + pl.kp + 64 + 127) & ~127}); };
    for (size_t i = 0; i < params.size(); i++) {
        const ParamDesc &d = params[i];
        want(d.seed_base + d.off_a);
        if (d.rows_k) want(d.seed_base + d.off_b);           // a vector's second seed is its first plus one: inside the margin
        if (!use.empty() && !use[i]) continue;
        if (!d.rows_k) {
            if (d.off_b != d.off_a + 1) { set_error("vector parameter with unrelated noise seeds"); return EGG_E_INVALID; }
            UpdVec v;
            const int x = d.seed_base + d.off_a + UPD_ORIGIN;
            v.len = d.cols_n; v.r = x & 15; v.x_a = x & ~15; v.lr_scale = d.lr_scale; v.model_off = d.model_off; v.opt_off = d.opt_off; v.ov = d.ov_in;
            pl.vecs.push_back(v);
        }
    }
    std::stable_sort(pl.vecs.begin(), pl.vecs.end(), [](const UpdVec &a, const UpdVec &b) { return a.len > b.len; });
    if (!pl.vecs.empty()) {
        pl.len_long = pl.vecs.front().len; pl.len_short = pl.vecs.back().len;
        for (const UpdVec &v : pl.vecs) {
            if (v.len == pl.len_long && pl.len_long != pl.len_short) pl.vec_long++;
            else if (v.len != pl.len_short) { set_error("vector parameters of more than two lengths"); return EGG_E_INVALID; }
        }
    }
    // the vectors' windows in blocks of 64 columns; tiles of eight vectors, up to 64 tiles
    if (pl.vecs.size() > 512) { set_error("%zu vector parameters: the vote product takes 512", pl.vecs.size()); return EGG_E_INVALID; }
    if (!pl.vecs.empty()) {
        std::stable_sort(pl.vecs.begin(), pl.vecs.end(), [](const UpdVec &a, const UpdVec &b) { return a.len != b.len ? a.len > b.len : a.x_a + a.r < b.x_a + b.r; });
        pl.vec_pad = ((int)pl.vecs.size() + 7) / 8 * 8;
        std::map<int, UpdVecCols> cover;
        for (size_t v = 0; v < pl.vecs.size(); v++) {
            const int x = pl.vecs[v].x_a + pl.vecs[v].r;
            for (int c = x & ~63; c < x + pairs; c += 64) {
                UpdVecCols &e = cover.emplace(c, UpdVecCols{c, {0, 0}}).first->second;
                e.tiles[v >> 8] |= 1u << ((v >> 3) & 31);
            }
        }
        for (const auto &e : cover) pl.vcols.push_back(e.second);
    }
    // batches in parameter order
    UpdBatch b;
    auto fresh = [&]() { memset(&b, 0, sizeof(b)); b.first = (int)pl.mats.size(); };
    auto close = [&]() {
        if (!b.count) return;
        // splits of the contraction: fewest k-blocks on the busiest SM, counting six for a work item's epilogue
        const int num_kb = pl.kp / UV_BK;
        int64_t best = -1;
        for (int s = 1; s <= 16 && s <= num_kb; s++) {
            const int per = (num_kb + s - 1) / s;
            if ((num_kb + per - 1) / per != s) continue;     // no empty split
            if (b.votes * s > std::max<int64_t>(UPD_VOTE_ELEMS, b.votes)) break;
            const int64_t waves = ((int64_t)b.tiles * s + num_sms / pl.cg - 1) / (num_sms / pl.cg), cost = waves * (per + 6) * 16 + s;
            if (best < 0 || cost < best) { best = cost; b.splits = s; }
        }
        pl.fn_bytes = std::max(pl.fn_bytes, (int64_t)std::max(b.fn_rows[0], b.fn_rows[1]) * pl.kp);
        pl.votes_elems = std::max(pl.votes_elems, b.votes * b.splits);
        pl.batches.push_back(b);
    };
    fresh();
    for (size_t i = 0; i < params.size(); i++) {
        const ParamDesc &d = params[i];
        if (!d.rows_k || (!use.empty() && !use[i])) continue;
        UpdMat m;
        memset(&m, 0, sizeof(m));
        m.rows_k = d.rows_k; m.cols_n = d.cols_n;
        const int fr = std::min(d.cols_n, d.rows_k);
        const int64_t wts = (int64_t)d.rows_k * d.cols_n;
        if (b.count && (b.count == UV_MAX_MATS || (int64_t)(b.fn_rows[0] + fr) * pl.kp > UPD_FN_BYTES || b.votes + wts > UPD_VOTE_ELEMS)) { close(); fresh(); }
        const int s_n = d.seed_base + d.off_a + UPD_ORIGIN, s_k = d.seed_base + d.off_b + UPD_ORIGIN;
        for (int form = 0; form < 2; form++) {
            UpdForm &f = m.form[form];
            f.fn_is_n = form || d.cols_n <= d.rows_k;
            const int s_tab = f.fn_is_n ? s_k : s_n, s_fn = f.fn_is_n ? s_n : s_k;
            f.r = s_tab & 15; f.x_tab = s_tab & ~15; f.x_fn = s_fn - f.r;
            f.fn_row0 = b.fn_rows[form];
            b.fn_rows[form] += f.fn_is_n ? d.cols_n : d.rows_k;
        }
        m.tile0 = b.tiles; m.tiles_n = (d.rows_k + UV_BN - 1) / UV_BN; m.blk0 = b.blocks; m.muon = d.muon;
        m.lr_scale = d.lr_scale; m.model_off = d.model_off; m.opt_off = d.opt_off; m.shadow_off = d.shadow_off; m.votes_off = b.votes;
        m.ov_in = d.ov_in; m.ov_out = d.ov_out;
        b.tiles += (d.cols_n + pl.cg * UV_BM - 1) / (pl.cg * UV_BM) * m.tiles_n; b.blocks += d.cols_n / 32 * (d.rows_k / 128); b.votes += wts; b.count++;
        b.any_adam |= !d.muon;
        pl.mats.push_back(m);
        pl.mat_param.push_back((int)i);
    }
    close();
    for (size_t bi = 0; bi < pl.batches.size(); bi++)
        for (int slot = 0; slot < 3; slot++) {               // square, wide, tall
            MuonGroup g = {(int)bi, 0, 0, (int)pl.list.size(), 0, slot};
            for (int i = pl.batches[bi].first; i < pl.batches[bi].first + pl.batches[bi].count; i++) {
                const UpdMat &m = pl.mats[i];
                if (!m.muon || (m.rows_k == m.cols_n ? 0 : (m.rows_k < m.cols_n ? 1 : 2)) != slot) continue;
                if (g.count && (m.rows_k != g.rows || m.cols_n != g.cols)) { set_error("Muon matrices of more than three shapes"); return EGG_E_INVALID; }
                g.rows = m.rows_k; g.cols = m.cols_n; g.count++;
                pl.list.push_back(i);
            }
            if (g.count) pl.groups.push_back(g);
        }
    std::sort(need.begin(), need.end());
    int end = 0, top = 0;
    for (const auto &n : need) {
        int c = std::max(n.first, end);
        top = std::max(top, n.second);
        for (; c < n.second; c += UPD_CHUNK) pl.chunks.push_back(make_int2(c, std::min(UPD_CHUNK, n.second - c)));
        end = std::max(end, n.second);
    }
    pl.pitch = top;
    auto image = [&](const void *v, size_t bytes) {
        const int64_t at = (int64_t)((pl.descriptors.size() + 255) & ~(size_t)255);
        pl.descriptors.resize((size_t)at + bytes);
        if (bytes) memcpy(pl.descriptors.data() + at, v, bytes);
        return at;
    };
    image(pl.mats.data(), pl.mats.size() * sizeof(UpdMat));
    pl.o_vecs = image(pl.vecs.data(), pl.vecs.size() * sizeof(UpdVec));
    pl.o_chunks = image(pl.chunks.data(), pl.chunks.size() * sizeof(int2));
    pl.o_list = image(pl.list.data(), pl.list.size() * sizeof(int));
    pl.o_vcols = image(pl.vcols.data(), pl.vcols.size() * sizeof(UpdVecCols));
    return EGG_OK;
}

}  // namespace egg
