// Row-owning int8 GEMM for sm_100a: the projections whose results pass through one of the reference's adaptive
// normalisations (adaptive_qkv_normalize / adaptive_layer_normalize, egg_adaptive_normalize.h:10-103) before anything
// else reads them.  Those normalisations need the abs-max of a WHOLE output row of H values, so one thread block
// keeps all H int32 accumulators of its 128 rows in tensor memory (H <= 512 = the 512 TMEM columns), finds the row
// maximum there and writes the requantised int8 row directly:
//
//   FUSED_QKV   q, k, v = AQN(rope(h.Wq + r1)), AQN(rope(h.Wk + r1)), AQN(h.Wv + r1)       (mgpu.cu:779-784)
//   FUSED_RES   x       = ALN(x + ((a.W + r1) >> shift) + bias + bias noise)                (mgpu.cu:746-756, 829-830)
//
// with r1 = ((Σ_k a_k b_k) * a_n * sign) >> (FIXED_POINT + SIGMA_SHIFT) (compute_linear_projection, mgpu.cu:553-572).
// A work unit is one 128-row tile of one part (q, k or v; the single part of FUSED_RES), made of H/BN sub-tiles of BN
// columns that occupy consecutive slots of a ring of 512/BN TMEM slots.  Roles: warp 0 feeds a shared-memory ring by
// TMA, warp 1 issues tcgen05.mma kind::i8, warps 2..17 are the epilogue (4 TMEM lane quarters x 4 column quarters;
// lane = row).  Per unit the epilogue makes two passes over tensor memory:
//   pass 1 (per sub-tile, as soon as its MMAs are done): rank-1 term, RoPE / residual + bias, running abs-max per lane; the
//          values go back to the same TMEM columns (tcgen05.st).  The residual projections leave floats: their maximum is
//          then one three-input instruction per two values instead of a maximum and a minimum, residual bytes are added by
//          a dot product against a unit vector, and the two shifts become one where int32 provably holds the unshifted sum
//          (both projections together 3 % faster; for q, k, v the same change spilled registers and gained nothing);
//   the four warps that share a lane quarter exchange their maxima through shared memory (128-thread named barrier);
//   pass 2 (per sub-tile): requantise (aln_quant_f), pack, write the warp's 32 x BN/4 int8 box to shared memory, release
//          the TMEM slot to the MMA warp, store the box with one TMA store.
// So the MMAs of the next unit's first sub-tile overlap pass 2 of this unit's last, and no int32 intermediate ever
// reaches HBM.  When seq_len is a multiple of 128 a tile's rows belong to one population member; otherwise (MM, seq_len a
// multiple of 32) every lane quarter of 32 rows has its own member.  Tables are the warp's own (MM, and q, k, v in 128-column
// sub-tiles), else those of a column quarter, shared by its four warps and double-buffered across units.  With MM the sub-tiles are
// 128 wide unless the block owns exactly 256 columns, so that the tables fit beside the operands.
// At H 256, seq_len 32 (262 144 rows) this replaces a projection with int32 output and a requantising pass: q|k|v 332 -> 200 us.
// For long contractions and wide tiles two blocks of a cluster form 256 rows together (CG = 2, cta_group::2): an SM gets fewer bytes from
// L2 than a 128 x 256 tile needs at the tensor cores' rate; the rule and its figures stand at launch_gemm_fused.
// Operands come by plain loads, no multicast; only tcgen05.commit of a pair arrives on both blocks' barriers.  Every wait is bounded and
// a timeout makes all later waits fall through so that the block drains, frees its tensor memory and reports.
#pragma once

#include "egg_gemm.cuh"

#include <type_traits>

namespace egg {

enum FusedMode { FUSED_QKV = 0, FUSED_RES = 1, FUSED_RES_LN = 2 };

struct FusedParams {
    int M, H, K;                 // rows (multiple of 128), width of one part, contraction
    int cl;                      // thread blocks that share a unit's columns (1 or 2): each owns
                                 // H/cl <= 512 columns of the unit's rows and the row maxima are exchanged through the
                                 // peer's shared memory
    int pair;                    // pairs of blocks form 256 rows together (chosen by launch_gemm_fused)
    int parts;                   // 3 (q, k, v: B is [3H][K]) or 1
    int seq_len;                 // rows of one member: multiple of 32
    const int8_t *nt;            // per-pair noise table of this wave
    int64_t nt_stride;
    int nt_a_off;                // A-noise of part 0 (length H); part p at + p*H
    int nt_c_off;                // FUSED_RES: bias-noise deltas [2][H] (-1: none)
    const int32_t *xb;           // Σ_k a_k b_k per row and part: xb[r * xb_stride + part]
    int xb_stride;
    int rank1_shift, out_shift;
    int pow_t;                   // FUSED_RES: merged_shift(), filled by launch_gemm_fused
    int one;                     // 1 (filled by launch_gemm_fused): the multiplier of additions issued as multiply-adds
    int unit[4];                 // 1 << 8i (filled by launch_gemm_fused): a dot product takes its selector from the parameters, not from a register
    const int8_t *bias;          // FUSED_RES: [H] or null
    const int4 *rope_t;          // see rope_entry()
    int rope_bit;
    int64_t part_rows;           // row distance between the parts in the output tensor map
    int *err;
    FastDiv fd_h, fd_seq;            // H and seq_len as multiply-shift divisors (filled by launch_gemm_fused)
    // FUSED_RES_LN: the mean-abs norm that follows the block (apply_standard_norm, mgpu.cu:646-678) and the row dots of
    // the projections after it, computed from the requantised row while it is still in shared memory
    int nt_w_m, nt_b_m;          // perturbed gain / bias tables (int16 [2][H]) in the noise table
    int ndots, nt_dot[3];        // B-noise vectors of the following projections
    int8_t *h_out;               // [M][H] normalised rows
    int32_t *xb_out;             // [M][xb_out_stride] row dots, ADDED to (cleared by the caller)
    int xb_out_stride;
};

constexpr int FUSED_MAX_H = 512;

template <int BN, bool MM, int CG>
struct FusedSmem {
    static constexpr int ST = CG == 2 ? 4 : GEMM_STAGES;        // ring stages: half of B in each block of a pair leaves room for a fourth
    static constexpr int NS = 512 / BN;                 // TMEM slots = most sub-tiles a unit can have
    static constexpr int WIDE = (MM && BN == 256) ? 256 : FUSED_MAX_H;      // most columns of a block
    static constexpr int NB = WIDE / BN;                // boxes per warp
    static constexpr int BOX = 32 * (BN / 4);           // bytes of one warp's int8 box: 32 rows x BN/4 columns
    alignas(1024) uint8_t a[ST][GEMM_BM * GEMM_BK];
    alignas(1024) uint8_t b[ST][BN / CG * GEMM_BK];
    // per epilogue warp and sub-tile: residual bytes in (FUSED_RES), requantised bytes out
    alignas(1024) uint8_t box[GEMM_EPI_WARPS][NB][BOX];
    // Tables of a unit, widened to int32: the A-noise of a column quarter's columns and, for the residual projections, (bias +
    // bias-noise delta of the member's sign) << shift behind it.  One per warp; where those do not fit (residual projections whose tiles
    // belong to one member) one per column quarter, double-buffered across units.
    static constexpr int TC = WIDE / 4;                 // columns of a quarter
    alignas(16) int32_t tab[GEMM_EPI_WARPS * TC * (MM ? 2 : 1)];
    alignas(16) int32_t rowpart[2][4][GEMM_BM];         // per-row abs-max of each column quarter (double-buffered across units)
    alignas(16) int32_t peer_max[2][GEMM_BM];           // per-row abs-max of the peer block's columns (written by the peer)
    alignas(16) uint16_t rowsum[4][GEMM_BM];            // FUSED_RES_LN: per-row Σ|x| of each column quarter (<= 127 * 128 columns)
    alignas(16) int32_t peer_sum[2][GEMM_BM];           // ... and of the peer block's columns
    alignas(8) uint64_t xbar[2];                        // arrival of the peer's maxima, one barrier per unit parity
    uint64_t xbar2[2];                                  // arrival of the peer's sums
    alignas(8) uint64_t full[ST];
    uint64_t empty[ST];
    uint64_t tmem_full[NS];
    uint64_t tmem_empty[NS];
    uint64_t rbar[GEMM_EPI_WARPS][NB];                  // arrival of a residual box
    uint32_t tmem_base;
    volatile int abort_flag;
};

// tensor map of an int8 matrix in boxes of 64 columns x 32 rows, 64-byte swizzle (egg_gemm_inst.cu)
int box_map(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t cols);

// Waits for an mbarrier phase unless the block is already draining after a timeout; a timeout here starts the drain.
__device__ __forceinline__ void fused_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *err, int code) {
    if (*abort_flag) return;
    if (!ptx::mbar_wait(bar, parity, 1000000000ull)) {
        *abort_flag = 1;
        if (err) atomicCAS(err, 0, code);
    }
}

// Words of the next unit's tables, loaded a unit ahead.
struct FusedTabWords { int32_t a, b, d; };

// FORM: FUSED_RES: both shifts as one (see pass 1); FUSED_RES_LN: three row dots follow (else one)
template <int CG, int BN, int MODE, bool MM, bool FORM>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_fused_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_o, const __grid_constant__ CUtensorMap tmap_r, const FusedParams p) {
    extern __shared__ uint8_t smem_raw[];
    using Smem = FusedSmem<BN, MM, CG>;
    Smem &sm = *reinterpret_cast<Smem *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int NS = Smem::NS;
    constexpr int CW = BN / 4;                  // columns of a sub-tile that one epilogue warp owns
    constexpr int NCH = CW / 16;                // 16-column chunks per warp and sub-tile
    constexpr int ST = Smem::ST;
    constexpr uint32_t STAGE_BYTES = GEMM_BM * GEMM_BK + BN / CG * GEMM_BK;      // of one block
    constexpr bool RES = (MODE != FUSED_QKV);   // residual + bias projections (O, MLP down)
    constexpr bool LN = (MODE == FUSED_RES_LN); // ... followed in the same epilogue by the next mean-abs norm
    constexpr bool MERGE = (MODE == FUSED_RES) && FORM;
    constexpr int NDOTS = LN ? (FORM ? 3 : 1) : 0;

    chain_next();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Clusters are consecutive blocks.  CG == 2: ranks that differ in the last bit are a pair, two row tiles of the same columns.
    const int rank = (int)blockIdx.x % (p.cl * CG), crank = rank / CG, prow = rank % CG;       // share of the columns, row tile of the pair
    const int peer = rank ^ CG;                                     // the block with the other share of this block's rows
    const int H0 = p.cl > 1 ? (p.H / 128 + 1) / 2 * 128 : p.H;      // columns of a part that the first block owns: half, rounded up to 128
    const int HL = crank ? p.H - H0 : H0;                           // ... that this block owns
    const int cofs = crank ? H0 : 0;                                // first of them
    const int first_unit = (int)blockIdx.x / (p.cl * CG), unit_step = (int)gridDim.x / (p.cl * CG);      // the blocks of a cluster walk the same units
    const int NT = HL / BN;                                         // sub-tiles per unit, 1..NS
    const int tiles_m = p.M / GEMM_BM;
    const int num_units = (tiles_m + CG - 1) / CG * p.parts;
    // row tile of a unit: an odd last one is formed by both blocks of its pair, and the second keeps it to itself
    auto row_tile = [&](int u) { return CG == 2 ? min(u * 2 + prow, tiles_m - 1) : u; };
    const int num_kb = (p.K + GEMM_BK - 1) / GEMM_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) { ptx::mbar_init(&sm.full[s], 1); ptx::mbar_init(&sm.empty[s], 1); }
        for (int a = 0; a < NS; a++) { ptx::mbar_init(&sm.tmem_full[a], 1); ptx::mbar_init(&sm.tmem_empty[a], CG * GEMM_EPI_WARPS); }
        for (int w = 0; w < GEMM_EPI_WARPS; w++)
            for (int a = 0; a < Smem::NB; a++) ptx::mbar_init(&sm.rbar[w][a], 1);
        ptx::mbar_init(&sm.xbar[0], GEMM_EPI_THREADS / 4);       // the peer's first column quarter: one arrival per row
        ptx::mbar_init(&sm.xbar[1], GEMM_EPI_THREADS / 4);
        ptx::mbar_init(&sm.xbar2[0], GEMM_EPI_THREADS / 4);
        ptx::mbar_init(&sm.xbar2[1], GEMM_EPI_THREADS / 4);
        sm.abort_flag = 0;
        ptx::fence_barrier_init();
    }
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
    if (p.cl * CG > 1) ptx::cluster_sync_all();     // the peers' barriers exist before anything arrives on them
    chain_wait();
    const uint32_t tmem_base = sm.tmem_base;

    if (warp == 0) {
        // ===================== TMA producer =====================
        if (ptx::elect_one()) {
            ptx::prefetch_tmap(&tmap_a);
            ptx::prefetch_tmap(&tmap_b);
            uint32_t it = 0;
            const uint32_t full_s = CG == 2 ? ptx::mapa_u32(ptx::smem_u32(sm.full), (uint32_t)rank & ~1u) : 0u;      // of the even block
            for (int unit = first_unit; unit < num_units && !sm.abort_flag; unit += unit_step) {
                const int mt = unit / p.parts, part = unit - mt * p.parts;
                const int m0 = row_tile(mt) * GEMM_BM;
                for (int j = 0; j < NT; j++) {
                    const int n0 = part * p.H + cofs + j * BN + prow * (BN / CG);
                    for (int kb = 0; kb < num_kb; kb++, it++) {
                        const int s = it % ST;
                        const uint32_t ph = (it / ST) & 1;
                        fused_wait(&sm.empty[s], ph ^ 1, &sm.abort_flag, p.err, DEV_TIMEOUT_EMPTY);
                        if (sm.abort_flag) break;
                        if (CG == 2) {
                            if (prow == 0) ptx::mbar_arrive_expect_tx(&sm.full[s], 2 * STAGE_BYTES);       // both blocks' bytes
                            ptx::tma_load_2d_pair(sm.a[s], &tmap_a, full_s + 8 * s, kb * GEMM_BK, m0);
                            ptx::tma_load_2d_pair(sm.b[s], &tmap_b, full_s + 8 * s, kb * GEMM_BK, n0);
                        } else {
                            ptx::mbar_arrive_expect_tx(&sm.full[s], STAGE_BYTES);
                            ptx::tma_load_2d(sm.a[s], &tmap_a, &sm.full[s], kb * GEMM_BK, m0);
                            ptx::tma_load_2d(sm.b[s], &tmap_b, &sm.full[s], kb * GEMM_BK, n0);
                        }
                    }
                    if (sm.abort_flag) break;
                }
            }
            if (sm.abort_flag) {   // let copies already in flight land before the block tears down
                const uint64_t t0 = ptx::globaltimer();
                while (ptx::globaltimer() - t0 < 200000ull) { __nanosleep(1000); }
            }
        }
    } else if (warp == 1) {
        // ===================== MMA issuer =====================
        if (prow == 0 && ptx::elect_one()) {
            constexpr uint32_t idesc = ptx::make_idesc_i8(CG * GEMM_BM, BN);
            uint32_t it = 0, stc = 0;
            for (int unit = first_unit; unit < num_units && !sm.abort_flag; unit += unit_step) {
                for (int j = 0; j < NT && !sm.abort_flag; j++, stc++) {
                    const int slot = stc % NS;
                    const uint32_t sph = (stc / NS) & 1;
                    fused_wait(&sm.tmem_empty[slot], sph ^ 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_EMPTY);          // (a pair: both blocks' epilogues arrive)
                    if (sm.abort_flag) break;
                    ptx::tc_fence_after();
                    const uint32_t d_tmem = tmem_base + (uint32_t)(slot * BN);
                    for (int kb = 0; kb < num_kb; kb++, it++) {
                        const int s = it % ST;
                        const uint32_t ph = (it / ST) & 1;
                        fused_wait(&sm.full[s], ph, &sm.abort_flag, p.err, DEV_TIMEOUT_FULL);
                        if (sm.abort_flag) break;
                        ptx::tc_fence_after();
                        const uint64_t da = ptx::make_smem_desc_sw128(ptx::smem_u32(sm.a[s]));
                        const uint64_t db = ptx::make_smem_desc_sw128(ptx::smem_u32(sm.b[s]));
#pragma unroll
                        for (int k = 0; k < GEMM_BK / 32; k++) {
                            if (CG == 2) ptx::mma_i8_pair(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                            else ptx::mma_i8(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        }
                        if (CG == 2) ptx::mma_commit_pair(&sm.empty[s], (uint32_t)rank); else ptx::mma_commit(&sm.empty[s]);
                    }
                    if (!sm.abort_flag) {
                        if (CG == 2) ptx::mma_commit_pair(&sm.tmem_full[slot], (uint32_t)rank); else ptx::mma_commit(&sm.tmem_full[slot]);
                    }
                }
            }
        }
    } else {
        // ===================== epilogue (16 warps) =====================
        const int ew = warp - 2;                   // 0..15
        const int quarter = warp & 3;              // TMEM lane quarter this warp may read
        const int cq = ew >> 2;                    // column quarter of every sub-tile
        const int row_in_tile = quarter * 32 + lane;
        // A warp meets the four warps of its rows (maxima, sums) and, where the tables are not its own, the four of its columns.
        // Table items are 4 consecutive columns, one a lane.
        constexpr bool OWN = MM || (MODE == FUSED_QKV && BN == 128);      // tables of the warp's own
        const bool tab_mine = lane < NT * (CW / 4) && (OWN || quarter == 0);
        const int tn = lane / (CW / 4) * BN + cq * CW + lane % (CW / 4) * 4;       // first column of this lane's item in the block's share
        auto table = [&](int buf) { return sm.tab + (OWN ? ew * (RES ? 2 : 1) : 2 * (4 * buf + cq)) * Smem::TC; };
        const long long half_ulp = 1ll << (p.rope_bit - 1);
        // shared address of this lane's row inside a box, and the XOR that swizzles its 16-byte pieces (64-byte swizzle
        // for 64-byte rows; 32-byte rows are stored densely)
        const uint32_t row_ofs = (uint32_t)lane * (uint32_t)CW;
        const uint32_t swz = (BN == 256) ? (uint32_t)((lane >> 1) & 3) : 0u;
        uint32_t stc = 0;
        int ucount = 0;
        int pf_xb = 0;
        FusedTabWords nxt = {0, 0, 0};

        auto tab_load = [&](int unit, FusedTabWords &w) {
            if (!tab_mine) return;
            const int mt = unit / p.parts, part = unit - mt * p.parts;
            const int mem = fast_div(row_tile(mt) * GEMM_BM + (MM ? 32 * quarter : 0), p.fd_seq);
            const int8_t *base = p.nt + (int64_t)(mem >> 1) * p.nt_stride;
            const int n = cofs + tn;
            w.a = *reinterpret_cast<const int32_t *>(base + p.nt_a_off + part * p.H + n);
            w.b = 0; w.d = 0;
            if (RES) {
                if (p.bias) w.b = *reinterpret_cast<const int32_t *>(p.bias + n);
                if (p.nt_c_off >= 0) w.d = *reinterpret_cast<const int32_t *>(base + p.nt_c_off + (mem & 1) * p.H + n);
            }
        };
        auto tab_store = [&](int buf, const FusedTabWords &w) {
            if (!tab_mine) return;
            int32_t *t = table(buf) + 4 * lane;
            *reinterpret_cast<int4 *>(t) = make_int4((int)(int8_t)w.a, (int)(int8_t)(w.a >> 8), (int)(int8_t)(w.a >> 16), w.a >> 24);
            if (RES) {
                int v[4];
#pragma unroll
                for (int b = 0; b < 4; b++)      // pre-shifted so that the sum joins the rank-1 product before its shift
                    v[b] = ((int)(int8_t)(w.b >> (8 * b)) + (int)(int8_t)(w.d >> (8 * b))) << (p.out_shift + p.rank1_shift);
                *reinterpret_cast<int4 *>(t + Smem::TC) = make_int4(v[0], v[1], v[2], v[3]);
            }
        };
        auto resid_request = [&](int unit) {      // lane 0: residual boxes of a unit, one per sub-tile
            const int m0 = row_tile(unit / p.parts) * GEMM_BM;
            for (int j = 0; j < NT; j++) {
                ptx::mbar_arrive_expect_tx(&sm.rbar[ew][j], 32 * CW);
                ptx::tma_load_2d(sm.box[ew][j], &tmap_r, &sm.rbar[ew][j], cofs + j * BN + cq * CW, m0 + quarter * 32);
            }
        };

        const uint32_t tmem_empty_s = CG == 2 ? ptx::mapa_u32(ptx::smem_u32(sm.tmem_empty), (uint32_t)rank & ~1u) : 0u;      // of the even block
        const uint32_t peer_max_s = p.cl > 1 ? ptx::mapa_u32(ptx::smem_u32(&sm.peer_max[0][0]), (uint32_t)peer) : 0u;
        const uint32_t peer_bar_s = p.cl > 1 ? ptx::mapa_u32(ptx::smem_u32(&sm.xbar[0]), (uint32_t)peer) : 0u;
        const uint32_t peer_sum_s = (LN && p.cl > 1) ? ptx::mapa_u32(ptx::smem_u32(&sm.peer_sum[0][0]), (uint32_t)peer) : 0u;
        const uint32_t peer_bar2_s = (LN && p.cl > 1) ? ptx::mapa_u32(ptx::smem_u32(&sm.xbar2[0]), (uint32_t)peer) : 0u;
        for (int unit = first_unit; unit < num_units; unit += unit_step, ucount++) {
            const int mt = unit / p.parts, part = unit - mt * p.parts;
            const int m0 = row_tile(mt) * GEMM_BM;
            const bool live = CG == 1 || 2 * mt + prow < tiles_m;
            const int r = m0 + row_in_tile;
            const int mem = fast_div(m0 + (MM ? quarter * 32 : 0), p.fd_seq);       // member of this warp's rows
            const int sgn = mem & 1;
            const int tb = ucount & 1;
            if (ucount == 0) {
                tab_load(unit, nxt);
                if (!OWN) tab_store(0, nxt);
                pf_xb = p.xb[(int64_t)r * p.xb_stride + part];
                if (RES && lane == 0) resid_request(unit);
            }
            if (OWN) {
                __syncwarp();              // every lane has left the previous unit
                tab_store(0, nxt);
                __syncwarp();
            } else {
                ptx::named_bar_sync(6 + cq, 128);          // tables of this unit are published; the group has left the previous unit
            }
            const int xbs = sgn ? -pf_xb : pf_xb;
            const int nunit = unit + unit_step;
            if (nunit < num_units) {
                tab_load(nunit, nxt);
                const int nmt = nunit / p.parts;
                pf_xb = p.xb[(int64_t)(row_tile(nmt) * GEMM_BM + row_in_tile) * p.xb_stride + (nunit - nmt * p.parts)];
            }
            const uint32_t tab_s = ptx::smem_u32(table(tb));
            // this token's entries of the rotation table: a warp's columns start at the same place in a head whatever the sub-tile is
            const int4 *rope = rope_entry(p.rope_t, r - mem * p.seq_len) + 32 * (((cq * CW) & 63) >> 2);

            // ---------------- pass 1: values and row abs-max, written back to tensor memory ----------------
            float rmx = 0.0f;
            int imx = 0, imn = 0;
            auto pass1 = [&](auto rope_part) {
            constexpr bool ROPE = decltype(rope_part)::value;
            for (int j = 0; j < NT; j++) {
                const uint32_t st = stc + (uint32_t)j;
                const int slot = st % NS;
                fused_wait(&sm.tmem_full[slot], (st / NS) & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_TMEM_FULL);
                const uint32_t box_s = ptx::smem_u32(sm.box[ew][j]) + row_ofs;
                if (RES) fused_wait(&sm.rbar[ew][j], ucount & 1, &sm.abort_flag, p.err, DEV_TIMEOUT_FULL);
                __syncwarp();                           // lanes leave the waits at different times; the TMEM accesses are warp-wide
                ptx::tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slot * BN + cq * CW);
                const uint32_t a32_s = tab_s + (uint32_t)(4 * j * CW), bcs_s = a32_s + 4 * Smem::TC;
                uint32_t v[2][16];
                ptx::tmem_ld16(taddr, v[0]);
#pragma unroll
                for (int c = 0; c < NCH; c++) {
                    int4 cs[4];
                    if (ROPE) {
                        // the lanes of a warp are consecutive tokens of one member: every load below is one contiguous run
#pragma unroll
                        for (int q4 = 0; q4 < 4; q4++) cs[q4] = __ldg(rope + 32 * (4 * c + q4));
                    }
                    int4 rs4 = make_int4(0, 0, 0, 0);
                    if (RES) rs4 = ptx::lds_v4(box_s + (((uint32_t)c ^ swz) << 4));
                    uint32_t *vc = v[c & 1];
                    ptx::tmem_ld_wait16(vc);
                    if (c + 1 < NCH) {
                        ptx::tmem_st_wait();            // the store of chunk c-1 read the registers the next load overwrites
                        ptx::tmem_ld16(taddr + 16 * (c + 1), v[(c + 1) & 1]);
                    }
#pragma unroll
                    for (int q4 = 0; q4 < 4; q4++) {
                        const int col = 16 * c + 4 * q4;
                        const int4 an = ptx::lds_v4(a32_s + 4 * col);
                        int x0, x1, x2, x3;
                        if (RES) {
                            // ((acc + r1 + (b << s)) >> s) + residual with r1 = (xb*a) >> t: the bias joins the rank-1 product
                            // ((b << (s+t)) is a multiple of 2^t); floor((acc + floor(y / 2^t)) / 2^s) ==
                            // floor((acc * 2^t + y) / 2^(s+t)) saves a shift where acc * 2^t + y cannot leave int32
                            const int4 b4 = ptx::lds_v4(bcs_s + 4 * col);
                            const int32_t rs = q4 == 0 ? rs4.x : (q4 == 1 ? rs4.y : (q4 == 2 ? rs4.z : rs4.w));
                            if (MERGE) {
                                const int sh2 = p.rank1_shift + p.out_shift;
                                x0 = ((int)vc[4 * q4] * p.pow_t + (xbs * an.x + b4.x)) >> sh2;
                                x1 = ((int)vc[4 * q4 + 1] * p.pow_t + (xbs * an.y + b4.y)) >> sh2;
                                x2 = ((int)vc[4 * q4 + 2] * p.pow_t + (xbs * an.z + b4.z)) >> sh2;
                                x3 = ((int)vc[4 * q4 + 3] * p.pow_t + (xbs * an.w + b4.w)) >> sh2;
                            } else {
                                x0 = (((xbs * an.x + b4.x) >> p.rank1_shift) * p.one + (int)vc[4 * q4]) >> p.out_shift;
                                x1 = (((xbs * an.y + b4.y) >> p.rank1_shift) * p.one + (int)vc[4 * q4 + 1]) >> p.out_shift;
                                x2 = (((xbs * an.z + b4.z) >> p.rank1_shift) * p.one + (int)vc[4 * q4 + 2]) >> p.out_shift;
                                x3 = (((xbs * an.w + b4.w) >> p.rank1_shift) * p.one + (int)vc[4 * q4 + 3]) >> p.out_shift;
                            }
                            x0 = __dp4a(rs, p.unit[0], x0);
                            x1 = __dp4a(rs, p.unit[1], x1);
                            x2 = __dp4a(rs, p.unit[2], x2);
                            x3 = __dp4a(rs, p.unit[3], x3);
                        } else {
                            x0 = ((xbs * an.x) >> p.rank1_shift) * p.one + (int)vc[4 * q4];
                            x1 = ((xbs * an.y) >> p.rank1_shift) * p.one + (int)vc[4 * q4 + 1];
                            x2 = ((xbs * an.z) >> p.rank1_shift) * p.one + (int)vc[4 * q4 + 2];
                            x3 = ((xbs * an.w) >> p.rank1_shift) * p.one + (int)vc[4 * q4 + 3];
                        }
                        if (ROPE) {
                            // integer RoPE on adjacent (even, odd) columns (apply_rope_integer, mgpu.cu:624-644)
                            const int e0 = x0, o0 = x1, e1 = x2, o1 = x3;
                            x0 = ptx::shr64_lo(ptx::mad_wide(-o0, cs[q4].y, ptx::mad_wide(e0, cs[q4].x, half_ulp)), p.rope_bit);
                            x1 = ptx::shr64_lo(ptx::mad_wide(o0, cs[q4].x, ptx::mad_wide(e0, cs[q4].y, half_ulp)), p.rope_bit);
                            x2 = ptx::shr64_lo(ptx::mad_wide(-o1, cs[q4].w, ptx::mad_wide(e1, cs[q4].z, half_ulp)), p.rope_bit);
                            x3 = ptx::shr64_lo(ptx::mad_wide(o1, cs[q4].z, ptx::mad_wide(e1, cs[q4].w, half_ulp)), p.rope_bit);
                        }
                        if (RES) {
                            const float f0 = __int2float_rn(x0), f1 = __int2float_rn(x1), f2 = __int2float_rn(x2), f3 = __int2float_rn(x3);
                            rmx = ptx::max3_abs(ptx::max3_abs(rmx, f0, f1), f2, f3);
                            x0 = __float_as_int(f0); x1 = __float_as_int(f1); x2 = __float_as_int(f2); x3 = __float_as_int(f3);
                        } else {
                            imx = __vimax3_s32(__vimax3_s32(imx, x0, x1), x2, x3);      // abs-max as max(max, -min)
                            imn = __vimin3_s32(__vimin3_s32(imn, x0, x1), x2, x3);
                        }
                        vc[4 * q4] = (uint32_t)x0; vc[4 * q4 + 1] = (uint32_t)x1; vc[4 * q4 + 2] = (uint32_t)x2; vc[4 * q4 + 3] = (uint32_t)x3;
                    }
                    ptx::tmem_st16(taddr + 16 * c, vc);
                }
                ptx::tmem_st_wait();
            }
            };
            if (MODE == FUSED_QKV && part < 2) pass1(std::integral_constant<bool, MODE == FUSED_QKV>());
            else pass1(std::integral_constant<bool, false>());
            sm.rowpart[tb][cq][row_in_tile] = RES ? __float_as_int(rmx) : max(imx, -imn);         // non-negative floats order like their bit patterns
            ptx::named_bar_sync(2 + quarter, 128);            // the four column quarters of this lane quarter
            int row_max = max(max(sm.rowpart[tb][0][row_in_tile], sm.rowpart[tb][1][row_in_tile]),
                              max(sm.rowpart[tb][2][row_in_tile], sm.rowpart[tb][3][row_in_tile]));
            if (p.cl > 1) {
                // the other half of the row lives in the peer block: its first column quarter writes the maximum of its
                // columns into this block's peer_max and arrives (release, cluster scope) on this block's barrier, and
                // vice versa.  Buffers and barriers alternate with the unit parity: the peer cannot get past this
                // exchange of unit u+1 before this block has arrived for it, that is after it has read unit u's value.
                if (cq == 0) {
                    ptx::st_cluster_u32(peer_max_s + (uint32_t)(tb * GEMM_BM + row_in_tile) * 4u, (uint32_t)row_max);
                    ptx::mbar_arrive_cluster(peer_bar_s + (uint32_t)tb * 8u);
                }
                if (!sm.abort_flag && !ptx::mbar_wait_cluster(&sm.xbar[tb], (uint32_t)(ucount >> 1) & 1u, 1000000000ull)) {
                    sm.abort_flag = 1;
                    if (p.err) atomicCAS(p.err, 0, DEV_TIMEOUT_PEER);
                }
                row_max = max(row_max, sm.peer_max[tb][row_in_tile]);
            }
            const float scale = RES ? 127.0f / (__int_as_float(row_max) + 1e-9f) : aln_scale(row_max);        // the same value either way

            // ---------------- pass 2: requantise, pack, store ----------------
            auto val = [](uint32_t w) { return RES ? __uint_as_float(w) : __int2float_rn((int)w); };
            int tot = 0;                                      // FUSED_RES_LN: Σ|x| over this warp's columns of the row
            for (int j = 0; j < NT; j++) {
                const uint32_t st = stc + (uint32_t)j;
                const int slot = st % NS;
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slot * BN + cq * CW);
                const uint32_t box_s = ptx::smem_u32(sm.box[ew][j]) + row_ofs;
                if (MODE == FUSED_QKV) {
                    // the store that last read this box was issued NT stores ago
                    if (lane == 0) { if (BN == 256 && NT == 2) ptx::tma_store_wait_read<1>(); else ptx::tma_store_wait_read<0>(); }
                    __syncwarp();
                }
                uint32_t v[2][16];
                ptx::tmem_ld16(taddr, v[0]);
#pragma unroll
                for (int c = 0; c < NCH; c++) {
                    uint32_t *vc = v[c & 1];
                    ptx::tmem_ld_wait16(vc);
                    if (c + 1 < NCH) ptx::tmem_ld16(taddr + 16 * (c + 1), v[(c + 1) & 1]);
                    uint32_t w[4];
#pragma unroll
                    for (int q4 = 0; q4 < 4; q4++)
                        w[q4] = ptx::pack_sat_s8(aln_quant_f(val(vc[4 * q4]), scale), aln_quant_f(val(vc[4 * q4 + 1]), scale),
                                                 aln_quant_f(val(vc[4 * q4 + 2]), scale), aln_quant_f(val(vc[4 * q4 + 3]), scale));
                    if (LN) {
#pragma unroll
                        for (int q4 = 0; q4 < 4; q4++) tot = abs_sum4(w[q4], tot);
                    }
                    ptx::sts_v4(box_s + (((uint32_t)c ^ swz) << 4), make_int4((int)w[0], (int)w[1], (int)w[2], (int)w[3]));
                }
                // this warp has read its part of the slot: hand it back to the MMA warp
                ptx::tc_fence_before();
                ptx::fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    if (CG == 2) ptx::mbar_arrive_peer(tmem_empty_s + 8 * slot); else ptx::mbar_arrive(&sm.tmem_empty[slot]);
                    if (live) ptx::tma_store_2d(&tmap_o, sm.box[ew][j], cofs + j * BN + cq * CW, (int)(part * p.part_rows) + m0 + quarter * 32);
                    ptx::tma_store_commit();
                }
            }
            stc += (uint32_t)NT;
            if (LN) {
                // ---------------- the mean-abs norm of the finished row (apply_standard_norm, mgpu.cu:646-678) ----------------
                // y = clip((x * w') / mean|x| + b'), and the dots of y with the B-noise of the projections that read it.  The
                // row's bytes are still in this lane's boxes; TMEM has been handed back, so the next unit's MMAs run meanwhile.
                sm.rowsum[cq][row_in_tile] = (uint16_t)tot;
                ptx::named_bar_sync(2 + quarter, 128);           // the sums of the four column quarters
                int total = (int)sm.rowsum[0][row_in_tile] + (int)sm.rowsum[1][row_in_tile] + (int)sm.rowsum[2][row_in_tile] + (int)sm.rowsum[3][row_in_tile];
                if (p.cl > 1) {      // the peer block's half of the row: same exchange as for the maxima
                    if (cq == 0) {
                        ptx::st_cluster_u32(peer_sum_s + (uint32_t)(tb * GEMM_BM + row_in_tile) * 4u, (uint32_t)total);
                        ptx::mbar_arrive_cluster(peer_bar2_s + (uint32_t)tb * 8u);
                    }
                    if (!sm.abort_flag && !ptx::mbar_wait_cluster(&sm.xbar2[tb], (uint32_t)(ucount >> 1) & 1u, 1000000000ull)) {
                        sm.abort_flag = 1;
                        if (p.err) atomicCAS(p.err, 0, DEV_TIMEOUT_PEER);
                    }
                    total += sm.peer_sum[tb][row_in_tile];
                }
                int mn = fast_div(total, p.fd_h);
                if (!mn) mn = 1;
                const float rinv = c_rinv_up.v[mn & 127];        // mn <= 127: a mean of absolute values of int8
                // From here a lane has 16 columns of several rows instead of a row: their gains, biases and noise are loaded once a
                // sub-tile, and a store covers whole rows of the box.  (A row a lane: four uniform 16-byte table reads per 16
                // columns, and stores of 16 bytes to 32 rows each; together they took the shared-memory port a seventh of the time.)
                constexpr int CPR = CW / 16, RPI = 32 / CPR;           // 16-byte pieces of a box row; rows of one step
                const int pc = lane % CPR, rr = lane / CPR;
                const int8_t *base = p.nt + (int64_t)(mem >> 1) * p.nt_stride;
                const int16_t *gain = reinterpret_cast<const int16_t *>(base + p.nt_w_m) + sgn * p.H + cofs, *shift = reinterpret_cast<const int16_t *>(base + p.nt_b_m) + sgn * p.H + cofs;
                int8_t *hrow = p.h_out + (int64_t)(m0 + quarter * 32 + rr) * p.H + cofs;
                int dot[CPR][NDOTS > 0 ? NDOTS : 1];
#pragma unroll
                for (int it = 0; it < CPR; it++)
#pragma unroll
                    for (int q = 0; q < NDOTS; q++) dot[it][q] = 0;
                for (int j = 0; j < NT; j++) {
                    const uint32_t box_s = ptx::smem_u32(sm.box[ew][j]);
                    const int col = j * BN + cq * CW + 16 * pc;
                    int w[8], b[8], d[NDOTS > 0 ? NDOTS : 1][4];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int4 wv = *reinterpret_cast<const int4 *>(gain + col + 8 * h), bv = *reinterpret_cast<const int4 *>(shift + col + 8 * h);
                        w[4 * h] = wv.x; w[4 * h + 1] = wv.y; w[4 * h + 2] = wv.z; w[4 * h + 3] = wv.w;
                        b[4 * h] = bv.x; b[4 * h + 1] = bv.y; b[4 * h + 2] = bv.z; b[4 * h + 3] = bv.w;
                    }
#pragma unroll
                    for (int q = 0; q < NDOTS; q++) {
                        const int4 dv = *reinterpret_cast<const int4 *>(base + p.nt_dot[q] + cofs + col);
                        d[q][0] = dv.x; d[q][1] = dv.y; d[q][2] = dv.z; d[q][3] = dv.w;
                    }
#pragma unroll
                    for (int it = 0; it < CPR; it++) {
                        const int row = it * RPI + rr;
                        const float ri = __shfl_sync(0xFFFFFFFFu, rinv, row);
                        const int4 xw = ptx::lds_v4(box_s + (uint32_t)row * CW + (((uint32_t)pc ^ (BN == 256 ? (uint32_t)((row >> 1) & 3) : 0u)) << 4));
                        uint32_t yw[4];
#pragma unroll
                        for (int q4 = 0; q4 < 4; q4++) {
                            const int xv = q4 == 0 ? xw.x : (q4 == 1 ? xw.y : (q4 == 2 ? xw.z : xw.w));
                            // x_i * w_i without widening either: a two-term dot product of the int16 pair with the word whose
                            // other byte is masked to zero, started from the bit pattern of 1.5 * 2^23 (i2f_small's addend);
                            // "+ b_i" the same way against a constant 1
                            const float f0 = __int_as_float(__dp2a_lo(w[2 * q4], xv & 0x000000FF, kMagicBits)) - kMagic;
                            const float f1 = __int_as_float(__dp2a_lo(w[2 * q4], xv & 0x0000FF00, kMagicBits)) - kMagic;
                            const float f2 = __int_as_float(__dp2a_hi(w[2 * q4 + 1], xv & 0x00FF0000, kMagicBits)) - kMagic;
                            const float f3 = __int_as_float(__dp2a_hi(w[2 * q4 + 1], xv & (int)0xFF000000, kMagicBits)) - kMagic;
                            const int y0 = __dp2a_lo(b[2 * q4], p.unit[0], __float2int_rz(f0 * ri));
                            const int y1 = __dp2a_lo(b[2 * q4], p.unit[1], __float2int_rz(f1 * ri));
                            const int y2 = __dp2a_lo(b[2 * q4 + 1], p.unit[0], __float2int_rz(f2 * ri));
                            const int y3 = __dp2a_lo(b[2 * q4 + 1], p.unit[1], __float2int_rz(f3 * ri));
                            yw[q4] = pack_clip8(y0, y1, y2, y3);
#pragma unroll
                            for (int q = 0; q < NDOTS; q++) dot[it][q] = __dp4a((int)yw[q4], d[q][q4], dot[it][q]);
                        }
                        if (live) *reinterpret_cast<int4 *>(hrow + (int64_t)(it * RPI) * p.H + col) = make_int4((int)yw[0], (int)yw[1], (int)yw[2], (int)yw[3]);
                    }
                }
                // the pieces of a row are neighbouring lanes: each keeps half of its rows and hands the others on, until lane pc of a
                // row group holds the whole sum of row pc * RPI + rr
#pragma unroll
                for (int q = 0; q < NDOTS; q++) {
                    if (CPR == 4) {
                        const bool up = pc & 2;
                        const int o0 = __shfl_xor_sync(0xFFFFFFFFu, up ? dot[0][q] : dot[2 % CPR][q], 2), o1 = __shfl_xor_sync(0xFFFFFFFFu, up ? dot[1][q] : dot[3 % CPR][q], 2);
                        dot[0][q] = (up ? dot[2 % CPR][q] : dot[0][q]) + o0;
                        dot[1][q] = (up ? dot[3 % CPR][q] : dot[1][q]) + o1;
                    }
                    const bool odd = pc & 1;
                    const int o = __shfl_xor_sync(0xFFFFFFFFu, odd ? dot[0][q] : dot[1][q], 1);
                    // every warp (and both blocks of a pair) adds its columns' share: integer sums, any order
                    if (live) atomicAdd(p.xb_out + (int64_t)(m0 + quarter * 32 + pc * RPI + rr) * p.xb_out_stride + q, (odd ? dot[1][q] : dot[0][q]) + o);
                }
                __syncwarp();          // all lanes have read their boxes before lane 0 lets the next residual bytes in
            }
            if (RES && lane == 0 && nunit < num_units) {
                // the boxes are free once their stores have read them: fetch the next unit's residual bytes
                ptx::tma_store_wait_read<0>();
                resid_request(nunit);
            }
            if (!OWN && nunit < num_units) tab_store(tb ^ 1, nxt);      // published by the next unit's barrier
        }
        if (lane == 0) ptx::tma_store_wait_all<0>();     // boxes still being copied out must land before the block retires
        if (sm.abort_flag) {   // draining after a timeout: residual boxes may still be in flight towards this block
            const uint64_t t0 = ptx::globaltimer();
            while (ptx::globaltimer() - t0 < 200000ull) { __nanosleep(1000); }
        }
        __syncwarp();
    }

    ptx::tc_fence_before();
    __syncthreads();
    // a pair gives its tensor memory back together, after both blocks' reads
    if (CG == 2) ptx::cluster_sync_all();
    if (warp == 1) {
        ptx::tc_fence_after();
        if (CG == 2) ptx::tmem_dealloc_pair(tmem_base, 512); else ptx::tmem_dealloc(tmem_base, 512);
    }
    // no block of a cluster retires while another may still write its maxima into it
    if (p.cl * CG > 1) { __syncwarp(); ptx::cluster_sync_all(); }
}

template <int BN, bool MM, int CG>
constexpr size_t fused_smem_bytes() { return sizeof(FusedSmem<BN, MM, CG>) + 1024; }
static_assert(fused_smem_bytes<256, false, 1>() <= EGG_MAX_SMEM && fused_smem_bytes<128, false, 1>() <= EGG_MAX_SMEM && fused_smem_bytes<256, true, 1>() <= EGG_MAX_SMEM &&
                  fused_smem_bytes<128, true, 1>() <= EGG_MAX_SMEM && fused_smem_bytes<256, false, 2>() <= EGG_MAX_SMEM && fused_smem_bytes<128, false, 2>() <= EGG_MAX_SMEM &&
                  fused_smem_bytes<256, true, 2>() <= EGG_MAX_SMEM && fused_smem_bytes<128, true, 2>() <= EGG_MAX_SMEM, "fused GEMM shared memory exceeds the 227 KB a block may use");

}  // namespace egg
