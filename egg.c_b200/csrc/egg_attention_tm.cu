// Causal integer-softmax attention (compute_attention, mgpu.cu:787-825) with scores, weights and sums in tensor memory.
//
// A persistent block per SM takes (member, head) items, or two members at a time where a member has 64 rows.  Q, K and V rows
// arrive by TMA as they lie; nothing is transposed or staged by hand.  For each tile of 128 queries and each chunk of 128 keys:
//   scores   S = Q K^T          tcgen05.mma kind::i8 into one of two 128-column buffers
//   maximum  a lane owns a query row; the two warps of a tensor-memory lane quarter share the chunk's four 32-key blocks
//   weights  table[max - score] as three 7-bit limbs, packed four keys to a word and written over the scores: limb l of key
//            block j at columns 32j + 8l.  They are the A operand, read from tensor memory (M = 128 rows, four keys a column)
//   sums     O_l += P_l V       V as an MN-major B operand straight from its rows; sixteen columns of ones beside it give the
//            sums of the weights
//   output   trunc((O_0 + 2^7 O_1 + 2^14 O_2) / sum), by eight other warps: every limb sum is below 127 * 127 * 512 < 2^23
// No score or weight passes through shared memory and no worker holds accumulators.  The MMA warp runs one chunk ahead of the
// weights; the quotients of a tile are formed while the next tile's weights are.  Tiles of up to two chunks keep their scores
// between maximum and weights; longer ones (seq_len > 256) form them twice.
// Bound: the chain maximum -> weights -> sums of a tile and the instructions beside it (issue slots half busy); tensor memory has
// room for one tile's sums only (2 x 128 + 3 x 80 of 512 columns), so that tiles overlap by one stage.  Measured against a block
// per head with mma.sync and 96 accumulators a thread (attention_kernel), 262 144 rows, H 512: 256 tokens 525 -> 298 us; whole
// passes: 80 tokens (H 384) 2.45 -> 1.35 ms, 512 tokens (H 1024) 18.5 -> 12.5 ms.  Sixteen weight warps that also divide: 375 us;
// with a register split for 16-column double buffering: 338 us (a tensor-memory load is back after 45 cycles); with the products of a
// chunk in one piece instead of two: 309 us.
// Every wait is bounded; a timeout makes all later waits fall through.  No multicast.
#include "egg_kernels.cuh"
#include "egg_gemm_fused.cuh"

#include <limits.h>

namespace egg {

constexpr int ATM_WARPS = 8;                           // of either kind of worker: 4 tensor-memory lane quarters x 2
constexpr int ATM_THREADS = 32 * (2 + 2 * ATM_WARPS);      // warp 0 copies, warp 1 MMAs, 2-9 weights, 10-17 quotients
constexpr int ATM_O_COL = 256;                         // tensor memory: two score buffers | O_l (80 each: 64 dims and the sum)

struct AtmParams {
    AttnParams a;
    int items, heads, pack;        // items; heads of a member; members in an item
    int rows, tiles;               // rows of an item, tiles of 128 queries
    int stages, stage_bytes, copies;                 // copies: of the weight table
    uint32_t k256;                 // 256, a run-time value: a multiply-add where a constant would become a permute on the busier pipe
    int *err;
};

struct AtmSmem {                   // behind the 1024-byte aligned stages and the table
    alignas(16) int32_t rowmax[2][2][128];
    alignas(8) uint64_t full[4], empty[4];           // Q, K, V of an item
    uint64_t s_full[2], s_free[2], p_ready[2][2], pv_done, o_full, o_free;      // p_ready: key blocks 0 and 1, 2 and 3
    uint32_t tmem_base;
    volatile int abort_flag;
};

__device__ __forceinline__ void atm_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *err, int code) {
    if (ptx::mbar_try_wait(bar, parity)) return;
    fused_wait(bar, parity, abort_flag, err, code);
}
// K-major operand of 64-byte rows with the 64-byte swizzle, or the same rows as an MN-major one: 8-row groups 512 bytes apart;
// MN-major: columns 64 and up lie `next` bytes further on
__device__ __forceinline__ uint64_t atm_desc_sw64(uint32_t smem_addr, uint32_t next = 512) {
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | (uint64_t)(next >> 4) << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
constexpr uint32_t ATM_B_MN = 1u << 16;                // instruction descriptor: B is MN-major
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void atm_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ uint2 atm_entry(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

// Four quotients from float estimates alone.  An estimate is off by less than 2^-21 of itself (num's two conversions and their sum,
// den's conversion, the approximate reciprocal and the product: three ulps), so with the reciprocal moved 2^-20 up and down its
// truncations enclose the quotient: where both agree that is it.  Elsewhere, one output in some 20 000 and the rows whose weight
// all lies on one key, `differ` is set and the outputs are divided again with att_div_small.
__device__ __forceinline__ uint32_t atm_quotients(const uint32_t *p0, const uint32_t *p1, const uint32_t *p2, float up, float down, uint32_t &differ) {
    float n[4];
#pragma unroll
    for (int i = 0; i < 4; i++) n[i] = fmaf(__int2float_rn((int)p2[i] * 128 + (int)p1[i]), 128.0f, __int2float_rn((int)p0[i]));
    const uint32_t a = ptx::pack_sat_s8(__float2int_rz(n[0] * up), __float2int_rz(n[1] * up), __float2int_rz(n[2] * up), __float2int_rz(n[3] * up));
    const uint32_t b = ptx::pack_sat_s8(__float2int_rz(n[0] * down), __float2int_rz(n[1] * down), __float2int_rz(n[2] * down), __float2int_rz(n[3] * down));
    differ |= a ^ b;
    return a;
}

// S8: shift_attn is 8, the table index is byte 1 of the clamped score.  BRIEF: several members share a tile, of which only the
// diagonal blocks count.
template <bool S8, bool BRIEF>
__global__ void __launch_bounds__(ATM_THREADS, 1) attention_tm_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                                                                      const __grid_constant__ CUtensorMap tmap_v, const AtmParams p) {
    extern __shared__ uint8_t atm_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(atm_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ones = base + p.stages * p.stage_bytes;                                 // 2 KB of 0x01
    uint32_t *lut = reinterpret_cast<uint32_t *>(ones + 2048);
    AtmSmem &sm = *reinterpret_cast<AtmSmem *>(lut + 512 * p.copies);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    chain_next();
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) { ptx::mbar_init(&sm.full[s], 1); ptx::mbar_init(&sm.empty[s], 1); }
        for (int b = 0; b < 2; b++) { ptx::mbar_init(&sm.s_full[b], 1); ptx::mbar_init(&sm.s_free[b], ATM_WARPS); ptx::mbar_init(&sm.p_ready[b][0], ATM_WARPS); ptx::mbar_init(&sm.p_ready[b][1], ATM_WARPS); }
        ptx::mbar_init(&sm.pv_done, 1); ptx::mbar_init(&sm.o_full, 1); ptx::mbar_init(&sm.o_free, ATM_WARPS);
        sm.abort_flag = 0;
        ptx::fence_barrier_init();
    }
    if (warp == 1) {
        ptx::tmem_alloc(&sm.tmem_base, 512);
        ptx::tmem_relinquish();
    }
    // the weights as three 7-bit limbs {l0 | l1 << 16, l2}, from the farthest score (entry 0) to the maximum (entry 255); `copies`
    // of each, a copy per two banks
    for (int i = threadIdx.x; i < 256 * p.copies / 2; i += ATM_THREADS) {
        const uint32_t w = (uint32_t)p.a.exp_lut[255 - (i * 2) / p.copies];
        const uint2 v = make_uint2((w & 127u) | ((w >> 7) & 127u) << 16, w >> 14);
        reinterpret_cast<uint4 *>(lut)[i] = make_uint4(v.x, v.y, v.x, v.y);
    }
    if (threadIdx.x < 128) reinterpret_cast<uint4 *>(ones)[threadIdx.x] = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
    ptx::fence_proxy_async();
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    chain_wait();
    const uint32_t tmem = sm.tmem_base;
    const int op = p.rows * 64;                                       // bytes of one operand of an item

    if (warp == 0) {
        // ===================== Q, K, V rows =====================
        if (ptx::elect_one()) {
            ptx::prefetch_tmap(&tmap_q); ptx::prefetch_tmap(&tmap_k); ptx::prefetch_tmap(&tmap_v);
            uint32_t it = 0;
            for (int item = blockIdx.x; item < p.items && !sm.abort_flag; item += gridDim.x, it++) {
                const int s = it % p.stages;
                atm_wait(&sm.empty[s], ((it / p.stages) & 1) ^ 1, &sm.abort_flag, p.err, DEV_TIMEOUT_EMPTY);
                if (sm.abort_flag) break;
                const int x = item % p.heads * 64, y = item / p.heads * p.pack * p.a.row_stride;
                uint8_t *d = base + s * p.stage_bytes;
                ptx::mbar_arrive_expect_tx(&sm.full[s], 3 * op);
                for (int r = 0; r < p.rows; r += 32) {
                    ptx::tma_load_2d(d + r * 64, &tmap_q, &sm.full[s], x, y + r);
                    ptx::tma_load_2d(d + op + r * 64, &tmap_k, &sm.full[s], x, y + r);
                    ptx::tma_load_2d(d + 2 * op + r * 64, &tmap_v, &sm.full[s], x, y + r);
                }
            }
            if (sm.abort_flag) {   // let copies already in flight land before the block tears down
                const uint64_t t0 = ptx::globaltimer();
                while (ptx::globaltimer() - t0 < 200000ull) { __nanosleep(1000); }
            }
        }
    } else if (warp == 1) {
        // ===================== MMA issuer =====================
        if (ptx::elect_one()) {
            // What has to happen before a score buffer is written again: its weights multiplied, or its maxima taken.  One word per
            // buffer: V's address / 16 (14 bits) | key blocks << 14 | weights << 17 | first chunk of a tile << 18 | last << 19 |
            // (stage to release + 1) << 20 | in use << 23
            uint32_t held0 = 0, held1 = 0, n = 0;
            uint32_t phase = 0;              // parities of the next waits: bits 0, 1 p_ready, 2, 3 s_free, 4 pv_done, 5 o_free
            const uint32_t ones_s = ptx::smem_u32(ones);
            auto consume = [&](uint32_t b) {
                const uint32_t L = b ? held1 : held0;
                if (b) held1 = 0; else held0 = 0;
                if (!(L >> 17 & 1)) {
                    atm_wait(&sm.s_free[b], phase >> (2 + b) & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_EMPTY);
                    phase ^= 4u << b;
                    ptx::tc_fence_after();
                    return;
                }
                const uint32_t ready = phase >> b & 1;
                phase ^= 1u << b;
                if (L >> 18 & 1) {           // the last tile's sums have been read
                    atm_wait(&sm.o_free, (phase >> 5 & 1) ^ 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_EMPTY);
                    phase ^= 32u;
                }
                constexpr uint32_t i_pv = ptx::make_idesc_i8(128, 80) | ATM_B_MN;
                const int blocks = L >> 14 & 7;
                uint32_t v = (L & 0x3FFF) << 4, at = tmem + 128 * b, acc = (L >> 18 & 1) ^ 1;
                for (int j = 0; j < 4; j++, v += 2048, at += 32, acc = 1) {
                    if (!(j & 1)) {          // every worker has written its block of this pair: half of the products run beside the other half's weights
                        atm_wait(&sm.p_ready[b][j >> 1], ready, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_EMPTY);
                        if (sm.abort_flag) return;
                        ptx::tc_fence_after();
                    }
                    if (j >= blocks) continue;
                    const uint64_t dv = atm_desc_sw64(v, ones_s - v);      // dims 64..79 are the block of ones
#pragma unroll
                    for (uint32_t l = 0; l < 3; l++) atm_mma_ts(tmem + ATM_O_COL + 80 * l, at + 8 * l, dv, i_pv, acc);
                }
                if (L >> 19 & 1) ptx::mma_commit(&sm.o_full);
                if (L >> 20 & 7) ptx::mma_commit(&sm.empty[(L >> 20 & 7) - 1]);
                ptx::mma_commit(&sm.pv_done);
                atm_wait(&sm.pv_done, phase >> 4 & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_FULL);       // the buffer's weights have been read
                phase ^= 16u;
            };
            uint32_t it = 0;
            for (int item = blockIdx.x; item < p.items && !sm.abort_flag; item += gridDim.x, it++) {
                const int s = it % p.stages;
                const uint32_t q = ptx::smem_u32(base + s * p.stage_bytes), k = q + (uint32_t)op, v = k + (uint32_t)op;
                atm_wait(&sm.full[s], (it / p.stages) & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_FULL);
                ptx::tc_fence_after();
                for (int t = 0; t < p.tiles && !sm.abort_flag; t++) {
                    const int nc = t + 1, sweeps = nc > 2 ? 2 : 1;
                    for (int w = 0; w < sweeps; w++)
                        for (int c = 0; c < nc && !sm.abort_flag; c++, n++) {
                            const uint32_t b = n & 1;
                            if (b ? held1 : held0) consume(b);
                            if (sm.abort_flag) break;
                            const int keys = min(128, p.rows - 128 * c);
                            const uint64_t da = atm_desc_sw64(q + 8192u * (uint32_t)t), db = atm_desc_sw64(k + 8192u * (uint32_t)c);
                            const uint32_t idesc = ptx::make_idesc_i8(128, keys);
                            ptx::mma_i8(tmem + 128u * b, da, db, idesc, 0u);
                            ptx::mma_i8(tmem + 128u * b, da + 2, db + 2, idesc, 1u);          // 64 dims: two 32-byte steps
                            ptx::mma_commit(&sm.s_full[b]);
                            const bool weights = w == sweeps - 1, last = c + 1 == nc;
                            const uint32_t L = (v + 8192u * (uint32_t)c) >> 4 | (uint32_t)(keys / 32) << 14 | (uint32_t)weights << 17 | (uint32_t)(c == 0) << 18 |
                                               (uint32_t)last << 19 | (weights && last && t + 1 == p.tiles ? (uint32_t)(s + 1) << 20 : 0u) | 1u << 23;
                            if (b) held1 = L; else held0 = L;
                        }
                }
            }
            for (int i = 0; i < 2; i++, n++)
                if (((n & 1) ? held1 : held0) && !sm.abort_flag) consume(n & 1);
        }
    } else if (warp < 2 + ATM_WARPS) {
        // ===================== maxima and weights =====================
        const int quarter = warp & 3, half = (warp - 2) >> 2;     // tensor-memory lane quarter; key blocks half and half + 2 of every chunk
        const int row = quarter * 32 + lane, sh = p.a.shift_attn, SP = p.a.row_stride;
        const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
        const uint32_t t_base = ptx::smem_u32(lut) + 8u * (uint32_t)(lane & (p.copies - 1)), t_mul = (uint32_t)(8 * p.copies) << (S8 ? 8 : 0);
        const int first_block = BRIEF ? quarter & 2 : 0;          // first 32-key block of the diagonal chunk that this quarter's rows see
        // block j of the diagonal chunk: 0 not looked at, 1 whole, 2 up to the row's own key
        auto kind = [&](int j) { return j > quarter || j < first_block ? 0 : (j == quarter ? 2 : 1); };
        const int kind0 = kind(half), kind1 = kind(half + 2);
        uint32_t n = 0, tile_no = 0;
        for (int item = blockIdx.x; item < p.items; item += gridDim.x) {
            const int row_i = item / p.heads * p.pack * SP;
            for (int t = 0; t < p.tiles; t++, tile_no++) {
                const int nc = t + 1, tb = tile_no & 1;
                const bool mine = 128 * t + quarter * 32 < p.rows && (!BRIEF || row_i + quarter * 32 < p.a.members * SP);
                // ---- row maxima over the keys a row sees (mgpu.cu:795-802) ----
                int mx = INT_MIN;
                for (int c = 0; c < nc; c++) {
                    const uint32_t ln = n + (uint32_t)c, b = ln & 1;
                    atm_wait(&sm.s_full[b], (ln >> 1) & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_FULL);
                    __syncwarp();
                    ptx::tc_fence_after();
#pragma unroll 1
                    for (int u = 0; u < 2; u++) {
                        const int k = !mine ? 0 : (c < t ? 1 : (u ? kind1 : kind0));
                        if (k == 0) continue;
                        uint32_t v[32];
                        ptx::tmem_ld32(t_lane + 128 * b + 32 * half + 64 * u, v);
                        ptx::tmem_ld_wait32(v);
                        int m[4] = {mx, INT_MIN, INT_MIN, INT_MIN};          // four chains
                        if (k == 1) {
#pragma unroll
                            for (int i = 0; i < 32; i += 2) m[i / 2 & 3] = __vimax3_s32(m[i / 2 & 3], (int)v[i], (int)v[i + 1]);
                        } else {
                            int to = lane;
                            asm volatile("" : "+r"(to));             // (conditions held over the tiles cost registers that spill)
#pragma unroll
                            for (int i = 0; i < 32; i++)
                                if (i <= to) m[i & 3] = max(m[i & 3], (int)v[i]);
                        }
                        mx = max(max(m[0], m[1]), max(m[2], m[3]));
                    }
                    if (nc > 2) {
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(&sm.s_free[b]);
                    }
                }
                if (nc > 2) n += (uint32_t)nc;
                sm.rowmax[tb][half][row] = mx;
                ptx::named_bar_sync(2 + quarter, 64);
                mx = max(sm.rowmax[tb][0][row], sm.rowmax[tb][1][row]);
                const int i0 = (255 - (mx >> sh)) * (1 << sh);
                // ---- weights (mgpu.cu:804-816) over the scores ----
                for (int c = 0; c < nc; c++) {
                    const uint32_t ln = n + (uint32_t)c, b = ln & 1;
                    if (nc > 2) {
                        atm_wait(&sm.s_full[b], (ln >> 1) & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_FULL);
                        __syncwarp();
                    }
                    ptx::tc_fence_after();
#pragma unroll 1
                    for (int u = 0; u < 2; u++) {
                        if (mine) {
                            const int k = c < t ? 1 : (u ? kind1 : kind0);
                            const uint32_t at = t_lane + 128 * b + 32 * half + 64 * u;
                            uint32_t l[3][8];
                            if (k) {
                                uint32_t v[32];
                                ptx::tmem_ld32(at, v);
                                ptx::tmem_ld_wait32(v);
#pragma unroll
                                for (int h = 0; h < 4; h++) {
                                    uint2 w[8];                      // the look-ups of 8 keys before the first word is put together
#pragma unroll
                                    for (int i = 0; i < 8; i++) {
                                        // score + (255 - maximum) << sh, negative where the difference exceeds 255: entry 0
                                        const uint32_t x = (uint32_t)__viaddmax_s32((int)v[8 * h + i], i0, 0);
                                        w[i] = atm_entry(__dp4a(S8 ? x : x >> sh, t_mul, t_base));           // one byte of the index: a masked key's entry exists, too
                                    }
#pragma unroll
                                    for (int g = 0; g < 2; g++) {
                                        const uint2 *e = w + 4 * g;
                                        const uint32_t ab = e[1].x * p.k256 + e[0].x, cd = e[3].x * p.k256 + e[2].x;       // [a0 b0 a1 b1], [c0 d0 c1 d1]
                                        l[0][2 * h + g] = __byte_perm(ab, cd, 0x5410);
                                        l[1][2 * h + g] = __byte_perm(ab, cd, 0x7632);
                                        l[2][2 * h + g] = __byte_perm(e[1].y * p.k256 + e[0].y, e[3].y * p.k256 + e[2].y, 0x5410);
                                    }
                                }
                                if (k == 2) {                         // keys up to the row's own stay
                                    int lost = 24 - 8 * lane;                // bits that the first four keys' word loses
                                    asm volatile("" : "+r"(lost));       // (masks held over the tiles cost registers that spill)
#pragma unroll
                                    for (int g = 0; g < 8; g++) {
                                        const uint32_t m = __funnelshift_rc(0xFFFFFFFFu, 0u, max(lost + 32 * g, 0));
#pragma unroll
                                        for (int q = 0; q < 3; q++) l[q][g] &= m;
                                    }
                                }
                            } else {
#pragma unroll
                                for (int g = 0; g < 8; g++) l[0][g] = l[1][g] = l[2][g] = 0;
                            }
                            ptx::tmem_st8(at, l[0]); ptx::tmem_st8(at + 8, l[1]); ptx::tmem_st8(at + 16, l[2]);
                            ptx::tmem_st_wait();
                        }
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(&sm.p_ready[b][u]);
                    }
                }
                n += (uint32_t)nc;
            }
        }
    } else {
        // ===================== quotients =====================
        const int quarter = warp & 3, half = (warp - 2 - ATM_WARPS) >> 2;       // tensor-memory lane quarter; 32 of the 64 dims
        const int row = quarter * 32 + lane, SP = p.a.row_stride, S = p.a.seq_len, H = p.a.H;
        const uint32_t t_lane = tmem + ((uint32_t)(quarter * 32) << 16);
        uint32_t tile_no = 0;
        for (int item = blockIdx.x; item < p.items; item += gridDim.x) {
            const int mem0 = item / p.heads * p.pack, col = item % p.heads * 64 + half * 32;
            for (int t = 0; t < p.tiles; t++, tile_no++) {
                const int r = 128 * t + row;                       // row of the item
                const int sub = BRIEF ? r >> 6 : 0;
                const bool own = r < p.rows && r - sub * SP < S && mem0 + sub < p.a.members;
                const int grow = mem0 * SP + r;
                int4 nb[2];
#pragma unroll
                for (int u = 0; u < 2; u++)
                    nb[u] = own ? *reinterpret_cast<const int4 *>(p.a.nt + (int64_t)((mem0 + sub) >> 1) * p.a.nt_stride + p.a.nt_o_b + col + 16 * u) : make_int4(0, 0, 0, 0);
                atm_wait(&sm.o_full, tile_no & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_FULL);
                __syncwarp();
                ptx::tc_fence_after();
                if (__any_sync(0xFFFFFFFFu, own)) {
                    uint32_t s0 = ptx::tmem_ld1(t_lane + ATM_O_COL + 64), s1 = ptx::tmem_ld1(t_lane + ATM_O_COL + 144), s2 = ptx::tmem_ld1(t_lane + ATM_O_COL + 224);
                    const uint32_t at = t_lane + ATM_O_COL + (uint32_t)(half * 32);
                    float up = 0.0f, down = 0.0f;
                    uint32_t den = 1;
                    int dot = 0;
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        uint32_t x[3][16];
#pragma unroll
                        for (int l = 0; l < 3; l++) ptx::tmem_ld16(at + 80 * l + 16 * u, x[l]);
#pragma unroll
                        for (int l = 0; l < 3; l++) ptx::tmem_ld_wait16(x[l]);
                        if (u == 0) {
                            asm volatile("" : "+r"(s0), "+r"(s1), "+r"(s2));
                            const uint32_t tot = s0 + (s1 << 7) + (s2 << 14);
                            den = tot ? tot : 1;                    // (no weight at all: divide by 1, mgpu.cu:818)
                            float rden;
                            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rden) : "f"(__uint2float_rn(den)));
                            up = rden * (1.0f + 0x1p-20f); down = rden * (1.0f - 0x1p-20f);
                        }
                        uint32_t o[4], differ = 0;
#pragma unroll
                        for (int g = 0; g < 4; g++) o[g] = atm_quotients(x[0] + 4 * g, x[1] + 4 * g, x[2] + 4 * g, up, down, differ);
                        if (__any_sync(0xFFFFFFFFu, differ != 0 && own)) {
#pragma unroll
                            for (int g = 0; g < 4; g++) {
                                int k[4];
#pragma unroll
                                for (int i = 0; i < 4; i++) k[i] = att_div_small((int)x[0][4 * g + i], (int)x[1][4 * g + i], (int)x[2][4 * g + i], den, up);
                                o[g] = ptx::pack_sat_s8(k[0], k[1], k[2], k[3]);
                            }
                        }
                        if (own) *reinterpret_cast<uint4 *>(p.a.ao + (int64_t)grow * H + col + 16 * u) = make_uint4(o[0], o[1], o[2], o[3]);
                        dot = __dp4a((int)o[0], nb[u].x, __dp4a((int)o[1], nb[u].y, __dp4a((int)o[2], nb[u].z, __dp4a((int)o[3], nb[u].w, dot))));
                    }
                    if (own) atomicAdd(&p.a.xbo[grow], dot);
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&sm.o_free);
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, 512);
    }
}

// Members of 64 to 512 rows (limb sums below 2^23), a multiple of 32.  By length alone, measured with 2 to 16 384 members at H 128 to
// 1024, evaluations of two layers, against the same with the mma.sync kernels.  64 tokens (two members in a tile, half of its blocks off
// the diagonal): the kernel 0.64 to 0.99 of attention_warp_kernel's time, the evaluation 1 to 18 % shorter.  48 tokens (a quarter of
// the rows are padding besides): the kernel 0.72 to 1.0, but 1.01 to 1.13 between 1000 and 6200 heads (20.8 -> 22.9 us); started early
// it hides that: the evaluation is up to 15 % shorter below 1500 heads, and from there on between 4 % shorter and 0.6 % longer, by
// which runs of one side differ too.  From 80 tokens the kernel takes 0.50 to 1.0 of attention_kernel's time.  Not 32 rows: four
// members would share a tile, most of whose blocks are off the diagonal, and every quarter has a row that sees one key only and is
// divided twice (65 536 members, H 256: 7.1 ms against 6.95 in attention_warp_kernel).
bool attention_tm_supported(int seq_len, int row_stride) { return seq_len <= row_stride && row_stride % 32 == 0 && row_stride >= 64 && row_stride <= 512; }

int launch_attention_tm(cudaStream_t st, const AttnParams &a, int num_sms, int *err) {
    AtmParams p;
    p.a = a;
    if ((unsigned)p.a.shift_attn > 20u) p.a.shift_attn = 20;          // scores are below 2^20 in magnitude: larger shifts leave the same sign
    p.err = err;
    p.heads = a.H / 64;
    p.pack = a.row_stride == 64 ? 2 : 1;
    p.rows = p.pack * a.row_stride;
    p.tiles = (p.rows + 127) / 128;
    p.items = (a.members + p.pack - 1) / p.pack * p.heads;
    p.stage_bytes = (3 * p.rows * 64 + 1023) / 1024 * 1024;
    const int fixed = 1024 + 2048 + (int)sizeof(AtmSmem) + 16;
    const int limit = EGG_MAX_SMEM;
    p.copies = 2 * p.stage_bytes + 32 * 1024 + fixed <= limit ? 16 : 8;      // a copy per two banks where two stages fit beside them
    p.k256 = 256;
    p.stages = (limit - fixed - 2048 * p.copies) / p.stage_bytes;
    if (p.stages > 4) p.stages = 4;
    size_t smem = (size_t)fixed + 2048 * p.copies + (size_t)p.stages * p.stage_bytes;
    if (smem < 116 * 1024) smem = 116 * 1024;                         // no second block that allocates tensor memory beside this one
    CUtensorMap m[3];
    const int8_t *src[3] = {a.q, a.k, a.v};
    for (int i = 0; i < 3; i++) {
        int rc = box_map(&m[i], src[i], (uint64_t)a.members * a.row_stride, (uint64_t)a.H);
        if (rc) return rc;
    }
    const bool s8 = p.a.shift_attn == 8, brief = p.pack > 1;
    auto kern = s8 ? (brief ? attention_tm_kernel<true, true> : attention_tm_kernel<true, false>) : (brief ? attention_tm_kernel<false, true> : attention_tm_kernel<false, false>);
    static std::atomic<bool> configured[4][EGG_MAX_DEVICES] = {};
    EGG_CUDA(allow_all_smem(kern, configured[2 * s8 + brief]));
    EGG_CUDA(launch_chained(kern, (unsigned)(p.items < num_sms ? p.items : num_sms), ATM_THREADS, smem, st, m[0], m[1], m[2], p));
    return EGG_OK;
}

}  // namespace egg
