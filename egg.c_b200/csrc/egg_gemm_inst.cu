// Instantiations and host launcher of the tcgen05 int8 GEMM.
#include "egg_kernels.cuh"
#include "egg_gemm_fused.cuh"
#include "egg_muon.cuh"

#include <cudaTypedefs.h>

namespace egg {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;

template <int BN, int EPI, int RPL = 0, int CG = 1>
static int set_attr() {
    EGG_CUDA(cudaFuncSetAttribute(gemm_i8_kernel<BN, EPI, RPL, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem_bytes<BN, CG>()));
    return EGG_OK;
}

template <int EPI, int RPL = 0>
static int set_attr_both() {
    int rc = set_attr<128, EPI, RPL>();
    if (rc) return rc;
    return set_attr<256, EPI, RPL>();
}

template <int BN, int MODE, bool MM, bool FORM, int CG = 1>
static int set_attr_fused_one() {
    EGG_CUDA(cudaFuncSetAttribute(gemm_fused_kernel<CG, BN, MODE, MM, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem_bytes<BN, MM, CG>()));
    return EGG_OK;
}
template <int BN, bool MM>
static int set_attr_fused() {
    int rc;
    if constexpr (BN == 256 && !MM) {
        if ((rc = set_attr_fused_one<BN, FUSED_QKV, MM, false, 2>()) || (rc = set_attr_fused_one<BN, FUSED_RES, MM, false, 2>()) ||
            (rc = set_attr_fused_one<BN, FUSED_RES, MM, true, 2>())) return rc;
    }
    if ((rc = set_attr_fused_one<BN, FUSED_QKV, MM, false>())) return rc;
    if ((rc = set_attr_fused_one<BN, FUSED_RES, MM, false>())) return rc;
    if ((rc = set_attr_fused_one<BN, FUSED_RES, MM, true>())) return rc;
    if ((rc = set_attr_fused_one<BN, FUSED_RES_LN, MM, false>())) return rc;
    if ((rc = set_attr_fused_one<BN, FUSED_RES_LN, MM, true>())) return rc;
    if constexpr (BN == 128 || !MM) {
        if ((rc = set_attr_fused_one<BN, FUSED_RES_LN, MM, false, 2>()) || (rc = set_attr_fused_one<BN, FUSED_RES_LN, MM, true, 2>())) return rc;
    }
    return EGG_OK;
}

int gemm_init() {
    if (!g_encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        EGG_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
        if (!fn || qres != cudaDriverEntryPointSuccess) { set_error("cuTensorMapEncodeTiled is not available from this driver"); return EGG_E_CUDA; }
        g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    }
    static bool done[EGG_MAX_DEVICES] = {};
    bool &d = done[current_device_slot()];
    if (d) return EGG_OK;
    int rc;
    if ((rc = set_attr_both<EPI_CLIP8>())) return rc;
    if ((rc = set_attr_both<EPI_CLIP8, 1>())) return rc;
    if ((rc = set_attr_both<EPI_GELU>())) return rc;
    if ((rc = set_attr_both<EPI_PRE32>())) return rc;
    if ((rc = set_attr_both<EPI_QKV>())) return rc;
    if ((rc = set_attr_both<EPI_GELU, 1>())) return rc;
    if ((rc = set_attr<256, EPI_GELU, 1, 2>())) return rc;
    if ((rc = set_attr<256, EPI_CLIP8, 1, 2>())) return rc;
    if ((rc = set_attr<256, EPI_VOTE, 0, 2>())) return rc;
    if ((rc = set_attr_both<EPI_PRE32, 1>())) return rc;
    if ((rc = set_attr_both<EPI_QKV, 1>())) return rc;
    if ((rc = set_attr<256, EPI_HEAD>())) return rc;
    if ((rc = set_attr<256, EPI_HEAD, 1>())) return rc;
    if ((rc = set_attr<256, EPI_LOGITS>())) return rc;
    if ((rc = set_attr<256, EPI_LOGITS, 1>())) return rc;
    if ((rc = set_attr_both<EPI_VOTE>())) return rc;
    if ((rc = set_attr<256, EPI_NULL>())) return rc;
    if ((rc = set_attr_fused<256, false>())) return rc;
    if ((rc = set_attr_fused<128, false>())) return rc;
    if ((rc = set_attr_fused<256, true>())) return rc;
    if ((rc = set_attr_fused<128, true>())) return rc;
    d = true;
    return EGG_OK;
}

// [rows][k] int8 row-major; box = 128 (k) x box_rows, 128-byte swizzle, out-of-range reads give zeros.
static int make_tmap(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t k, uint32_t box_rows) {
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (k & 15)) { set_error("GEMM operand is not 16-byte aligned (ptr %p, k %llu)", ptr, (unsigned long long)k); return EGG_E_INVALID; }
    cuuint64_t gdim[2] = {k, rows};
    cuuint64_t gstride[1] = {k};
    cuuint32_t box[2] = {(cuuint32_t)GEMM_BK, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d) rows=%llu k=%llu box_rows=%u", (int)r, (unsigned long long)rows, (unsigned long long)k, box_rows); return EGG_E_CUDA; }
    return EGG_OK;
}

int upd_tensor_map(void *map, const void *ptr, uint64_t rows, uint64_t pitch, uint32_t box_rows) {
    if (!g_encode) { set_error("gemm_init() was not called"); return EGG_E_STATE; }
    return make_tmap(static_cast<CUtensorMap *>(map), ptr, rows, pitch, box_rows);
}

// [rows][cols] bf16 row-major; box = 64 columns x 128 rows, 128-byte swizzle
int bf16_tensor_map(void *map, const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    if (!g_encode) { set_error("gemm_init() was not called"); return EGG_E_STATE; }
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (cols & 7)) { set_error("bf16 operand is not 16-byte aligned (ptr %p, cols %llu)", ptr, (unsigned long long)cols); return EGG_E_INVALID; }
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols * 2};
    cuuint32_t box[2] = {64, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(static_cast<CUtensorMap *>(map), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (bf16) failed (%d) rows=%llu cols=%llu", (int)r, (unsigned long long)rows, (unsigned long long)cols); return EGG_E_CUDA; }
    return EGG_OK;
}

// [rows][cols] int32 row-major output written by TMA stores of 16-column x 32-row boxes (64-byte swizzle in shared memory)
static int make_tmap_out(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t cols) {
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (cols & 3)) { set_error("GEMM output is not 16-byte aligned (ptr %p, cols %llu)", ptr, (unsigned long long)cols); return EGG_E_INVALID; }
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols * 4};
    cuuint32_t box[2] = {16, 32};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void *>(ptr), gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (output) failed (%d) rows=%llu cols=%llu", (int)r, (unsigned long long)rows, (unsigned long long)cols); return EGG_E_CUDA; }
    return EGG_OK;
}

// [rows][cols] int8 row-major output written by TMA stores of 64-column x 32-row boxes (64-byte swizzle)
static int make_tmap_out8(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t cols) {
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (cols & 15)) { set_error("GEMM output is not 16-byte aligned (ptr %p, cols %llu)", ptr, (unsigned long long)cols); return EGG_E_INVALID; }
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols};
    cuuint32_t box[2] = {64, 32};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (int8 output) failed (%d) rows=%llu cols=%llu", (int)r, (unsigned long long)rows, (unsigned long long)cols); return EGG_E_CUDA; }
    return EGG_OK;
}

// [rows][cols] int8 row-major moved as box_cols-column x 32-row boxes: 64-byte rows swizzled (64-byte pattern), 32-byte
// rows stored densely
static int make_tmap_box8(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t cols, uint32_t box_cols) {
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (cols & 15) || (box_cols != 64 && box_cols != 32)) {
        set_error("int8 box map unsupported (ptr %p, cols %llu, box %u)", ptr, (unsigned long long)cols, box_cols);
        return EGG_E_INVALID;
    }
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstride[1] = {cols};
    cuuint32_t box[2] = {box_cols, 32};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), gdim, gstride, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (int8 boxes) failed (%d) rows=%llu cols=%llu", (int)r, (unsigned long long)rows, (unsigned long long)cols); return EGG_E_CUDA; }
    return EGG_OK;
}

int box_map(CUtensorMap *m, const void *ptr, uint64_t rows, uint64_t cols) {
    if (!g_encode) { set_error("gemm_init() was not called"); return EGG_E_STATE; }
    return make_tmap_box8(m, ptr, rows, cols, 64);
}

// Blocks that share a unit of the row-owning GEMM: one up to 512 columns, a cluster of two above (0: unsupported width).
// An odd multiple of 128 is shared unevenly (640 = 384 + 256, 896 = 512 + 384).
int fused_cluster_size(int hidden) {
    if (hidden <= 0 || hidden % 128) return 0;
    if (hidden <= FUSED_MAX_H) return 1;
    if (hidden <= 2 * FUSED_MAX_H) return 2;
    return 0;
}

template <int BN, int MODE, bool MM, bool FORM, int CG>
static int launch_fused_cg(cudaStream_t st, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &to, const CUtensorMap &tr,
                            const FusedParams &p, int units, int num_sms) {
    auto kern = gemm_fused_kernel<CG, BN, MODE, MM, FORM>;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = fused_smem_bytes<BN, MM, CG>();
    const int cluster = p.cl * CG;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int groups = num_sms / cluster;                  // resident blocks (clusters of blocks)
    if (cluster > 1) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;                  // (the occupancy question is about the cluster alone)
        // the clusters that can be resident at once (a GPC whose free SMs are no multiple leaves some out): asked once a size
        static std::atomic<int> max_dev[2][EGG_MAX_DEVICES] = {};
        std::atomic<int> &max_pairs = max_dev[p.cl > 1][current_device_slot()];
        if (max_pairs == 0) {
            cfg.gridDim = dim3((unsigned)(num_sms / cluster * cluster));
            int n = 0;
            EGG_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
            if (n < 1) { set_error("no cluster of blocks of the row-owning GEMM fits on the device"); return EGG_E_CUDA; }
            max_pairs = n;
        }
        if (groups > max_pairs) groups = max_pairs;
    }
    if (groups > units) groups = units;
    cfg.gridDim = dim3((unsigned)(groups * cluster));
    cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 1 : 0;
    if (t_chain) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    EGG_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, to, tr, p));
    return EGG_OK;
}

template <int BN, int MODE, bool MM, bool FORM = false>
static int launch_fused_one(cudaStream_t st, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &to, const CUtensorMap &tr,
                            const FusedParams &p, int units, int num_sms) {
    if constexpr (MODE == FUSED_RES_LN ? BN == 128 || !MM : BN == 256 && !MM) {
        if (p.pair) return launch_fused_cg<BN, MODE, MM, FORM, 2>(st, ta, tb, to, tr, p, units, num_sms);
    }
    return launch_fused_cg<BN, MODE, MM, FORM, 1>(st, ta, tb, to, tr, p, units, num_sms);
}

template <int BN, bool MM>
static int launch_fused_mode(cudaStream_t st, int mode, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &to, const CUtensorMap &tr,
                             const FusedParams &p, int units, int num_sms) {
    if (mode == FUSED_QKV) return launch_fused_one<BN, FUSED_QKV, MM>(st, ta, tb, to, tr, p, units, num_sms);
    if (mode == FUSED_RES_LN && p.ndots == 3) return launch_fused_one<BN, FUSED_RES_LN, MM, true>(st, ta, tb, to, tr, p, units, num_sms);
    if (mode == FUSED_RES_LN) return launch_fused_one<BN, FUSED_RES_LN, MM>(st, ta, tb, to, tr, p, units, num_sms);
    if (p.pow_t) return launch_fused_one<BN, FUSED_RES, MM, true>(st, ta, tb, to, tr, p, units, num_sms);
    return launch_fused_one<BN, FUSED_RES, MM>(st, ta, tb, to, tr, p, units, num_sms);
}

int launch_gemm_fused(cudaStream_t st, int mode, const int8_t *A, const int8_t *B, int8_t *out, const int8_t *resid,
                      const FusedParams &p_in, int num_sms) {
    FusedParams p = p_in;
    if (!g_encode) { set_error("gemm_init() was not called"); return EGG_E_STATE; }
    p.cl = fused_cluster_size(p.H);
    if (p.M <= 0 || p.M % GEMM_BM || p.seq_len % 32 || p.cl == 0 || p.K % 16 || p.parts < 1 ||
        (mode != FUSED_QKV && (p.parts != 1 || !resid)) || (mode != FUSED_QKV && mode != FUSED_RES && mode != FUSED_RES_LN) ||
        (mode == FUSED_RES_LN && (!p.h_out || !p.xb_out || (p.ndots != 1 && p.ndots != 3)))) {
        set_error("unsupported row-owning GEMM shape M=%d H=%d K=%d parts=%d seq_len=%d", p.M, p.H, p.K, p.parts, p.seq_len);
        return EGG_E_INVALID;
    }
    if (mode != FUSED_QKV && p.out_shift + p.rank1_shift > PRESHIFT_MAX) {
        set_error("shifts %d + %d too large for the pre-shifted bias table", p.out_shift, p.rank1_shift);
        return EGG_E_INVALID;
    }
    int units = (p.M / GEMM_BM) * p.parts;
    // few units: two blocks share each, so that a unit's products and its epilogue take half as long on SMs that would idle
    // (2048 rows, H 256: MLP-down 12.7 -> 11.3 us, Q|K|V 8.6 -> 7.2, output projection 7.4 -> 6.3)
    if (p.cl == 1 && p.H >= 256 && 2 * units <= num_sms) p.cl = 2;
    const int hl = p.H % (128 * p.cl) ? 128 : p.H / p.cl;      // columns per block (uneven shares: whole 128-column sub-tiles)
    const bool mm = p.seq_len % GEMM_BM != 0;        // a tile spans members: tables of the warp's own, see the kernel
    const int bn = (mm ? hl == 256 : hl % 256 == 0) ? 256 : 128;      // (128-column sub-tiles at H = 512 were measured: +30 % on MLP-down)
    // Pairs of blocks where the products wait for their operands: a 128 x 256 tile takes 96 bytes a clock at the tensor cores' rate and an SM
    // gets some 57, a pair's half needs 64.  The two blocks' epilogues wait for one another, so not where those are the longer part.
    // Down projection with the norm, per evaluation of 4 or 2 layers: K 2048 8.24 -> 7.01 ms, 2560 2.43 -> 2.17, 4096 3.49 -> 3.31, 1536 1.52 ->
    // 1.41, but 1024 2 to 4 % longer.  Q|K|V in tiles of one member and 256 columns, one block to a row: H 512 5.94 -> 5.48, H 256 2.84 -> 2.74;
    // output projection at H 512 5 % shorter, at H 256 as much longer.  Tiles of several members, narrower ones and rows of two
    // blocks: Q|K|V 2 to 12 % longer.  From two units an SM on, for clusters of four: the down projection of 148 and 222 row tiles 9 to 11 and 2 to 6 us
    // a launch longer (H 640 to 1024), of 296 up to 2 us shorter, of 592 17 to 32; Q|K|V at H 256 of 100 to 592 the same within 0.4 us.
    const bool wide = p.cl == 1 && bn == 256 && !mm;
    p.pair = units >= 2 * num_sms && (mode == FUSED_RES_LN ? p.K >= 1536 && (bn == 128 || !mm) : wide && (mode == FUSED_QKV || p.K >= 512));
    if (p.pair) units = (p.M / GEMM_BM + 1) / 2 * p.parts;
    p.fd_seq = make_fastdiv(p.seq_len);
    p.fd_h = make_fastdiv(p.H);
    p.one = 1;
    for (int i = 0; i < 4; i++) p.unit[i] = 1 << (8 * i);
    p.pow_t = mode == FUSED_RES ? merged_shift(p.K, p.rank1_shift, p.out_shift) : 0;
    CUtensorMap ta, tb, to, tr;
    int rc;
    if ((rc = make_tmap(&ta, A, (uint64_t)p.M, (uint64_t)p.K, GEMM_BM))) return rc;
    if ((rc = make_tmap(&tb, B, (uint64_t)p.parts * p.H, (uint64_t)p.K, (uint32_t)(p.pair ? bn / 2 : bn)))) return rc;
    const uint64_t out_rows = p.parts > 1 ? (uint64_t)p.parts * (uint64_t)p.part_rows : (uint64_t)p.M;
    if ((rc = make_tmap_box8(&to, out, out_rows, (uint64_t)p.H, (uint32_t)bn / 4))) return rc;
    tr = to;
    if (mode != FUSED_QKV && (rc = make_tmap_box8(&tr, resid, (uint64_t)p.M, (uint64_t)p.H, (uint32_t)bn / 4))) return rc;
    if (bn == 256) return mm ? launch_fused_mode<256, true>(st, mode, ta, tb, to, tr, p, units, num_sms) : launch_fused_mode<256, false>(st, mode, ta, tb, to, tr, p, units, num_sms);
    return mm ? launch_fused_mode<128, true>(st, mode, ta, tb, to, tr, p, units, num_sms) : launch_fused_mode<128, false>(st, mode, ta, tb, to, tr, p, units, num_sms);
}

template <int BN, int EPI, int RPL = 0>
static int launch_one(cudaStream_t st, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &to, const GemmParams &p, int num_sms) {
    int tiles = ((p.M + GEMM_BM - 1) / GEMM_BM) * (p.N / BN) * ((EPI == EPI_VOTE && p.k_splits > 1) ? p.k_splits : 1);
    int grid = tiles < num_sms ? tiles : num_sms;
    CUtensorMap tr = ta;       // residual bytes as 64-column x 32-row boxes (row-per-lane residual projections with BN = 256 only)
    if (EPI == EPI_PRE32 && RPL && BN == 256) {
        int rc = make_tmap_out8(&tr, p.resid, (uint64_t)p.M, (uint64_t)p.N);
        if (rc) return rc;
    }
    EGG_CUDA(launch_chained(gemm_i8_kernel<BN, EPI, RPL>, grid, GEMM_THREADS, gemm_smem_bytes<BN>(), st, ta, tb, to, tr, p));
    return EGG_OK;
}

// Pairs of blocks with the tiles of 256 columns of two row tiles.
template <int EPI, int RPL>
static int launch_pair(cudaStream_t st, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &to, const GemmParams &p, int num_sms) {
    auto kern = gemm_i8_kernel<256, EPI, RPL, 2>;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = gemm_smem_bytes<256, 2>();
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    static std::atomic<int> max_dev[EGG_MAX_DEVICES] = {};          // pairs that can be resident at once
    std::atomic<int> &most = max_dev[current_device_slot()];
    if (most == 0) {
        cfg.gridDim = dim3((unsigned)(num_sms / 2 * 2));
        int n = 0;
        EGG_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
        if (n < 1) { set_error("no pair of blocks of the GEMM fits on the device"); return EGG_E_CUDA; }
        most = n < num_sms / 2 ? n : num_sms / 2;
    }
    const int tiles = ((p.M + 2 * GEMM_BM - 1) / (2 * GEMM_BM)) * (p.N / 256) * ((EPI == EPI_VOTE && p.k_splits > 1) ? p.k_splits : 1);
    const int pairs = most;
    cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs)));
    if (t_chain) {
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    EGG_CUDA(cudaLaunchKernelEx(&cfg, kern, ta, tb, to, ta, p));
    return EGG_OK;
}

template <int EPI, int RPL = 0>
static int launch_bn(cudaStream_t st, int bn, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &to, const GemmParams &p, int num_sms) {
    if (bn == 256) return launch_one<256, EPI, RPL>(st, ta, tb, to, p, num_sms);
    return launch_one<128, EPI, RPL>(st, ta, tb, to, p, num_sms);
}

// evaluation epilogues whose rows come in whole 32-row groups per member take the row-per-lane form
template <int EPI>
static int launch_eval(cudaStream_t st, int bn, const CUtensorMap &ta, const CUtensorMap &tb, const CUtensorMap &to, const GemmParams &p, int num_sms) {
    if (p.seq_len % 32 == 0 && p.rpl >= 0) return launch_bn<EPI, 1>(st, bn, ta, tb, to, p, num_sms);
    return launch_bn<EPI, 0>(st, bn, ta, tb, to, p, num_sms);
}

// Whether pairs of blocks form the tiles of 256 columns (see launch_gemm_fused for what bounds them).  MLP-up: K 384 0.89 -> 0.87 ms,
// 512 5.75 -> 5.45, 640 1.23 -> 1.09, 768 1.70 -> 1.45, 896 2.22 -> 1.85, 1024 2.45 -> 1.99; projections of as many columns: 512 0.155 ->
// 0.146, 2048 0.52 -> 0.46, 4096 3.40 -> 2.92 (2.6 -> 3.0 int8 POP/s).  At K 256 between 2 % shorter and 1 % longer.
// Votes of one matrix: by the contraction of one item, which has to make up for a launch of clusters (whole calls of 40 to 60 us): up to 384
// 2 us longer, at 512 the same, above up to 10 % shorter (4096 x 4096 from 16 384 pairs 463 -> 415 us).
// Projections of their own (and the recurrent model's): the same launch against some (K - 256) / 150 ns a tile.  K 384 1.2 us longer up to 2368
// tiles, the same at 4736; 512 0.7 longer at 1184, 1.0 shorter at 1776 (85 us), 30 at 9472 (309); 768 1.5 longer at 592, 1.0 shorter at 888;
// 1024 0.9 shorter at 592 (58).  MLP-up stands in a chain of launches, where the clusters' cost does not show: K 384 and 512 the same from 592 tiles on.
static bool pairs_form(int epi, const GemmParams &p, int rows_m, int num_sms) {
    const int splits = epi == EPI_VOTE && p.k_splits > 1 ? p.k_splits : 1;
    const int64_t tiles = (int64_t)rows_m * (p.N / 256) * splits;
    if (epi == EPI_VOTE) return p.K > 512 * splits && rows_m % 2 == 0 && tiles >= num_sms;
    if (p.seq_len % 32 || p.rpl < 0 || p.K < 384 || tiles < 4 * num_sms) return false;
    return epi == EPI_GELU || (epi == EPI_CLIP8 && (p.K - 256) * tiles >= 2560 * num_sms);
}

int launch_gemm(cudaStream_t st, int epi, const int8_t *A, const int8_t *B, const GemmParams &p_in, int num_sms) {
    GemmParams p = p_in;
    if (!g_encode) { set_error("gemm_init() was not called"); return EGG_E_STATE; }
    if (p.M <= 0 || p.N % 128 || p.K % 16) { set_error("unsupported GEMM shape M=%d N=%d K=%d", p.M, p.N, p.K); return EGG_E_INVALID; }
    int bn = (p.N % 256 == 0) ? 256 : 128;
    // few tiles: half as wide, on twice as many SMs (2048 rows, H 256: MLP-up 7.0 -> 5.8 us)
    if (epi <= EPI_QKV && bn == 256 && 2 * ((p.M + GEMM_BM - 1) / GEMM_BM) * (p.N / 256) <= num_sms) bn = 128;
    if (epi == EPI_QKV && (p.third % bn)) bn = 128;
    if (epi == EPI_QKV && (p.third % 128)) { set_error("hidden_dim must be a multiple of 128"); return EGG_E_INVALID; }
    if (epi == EPI_HEAD && p.N != 256) { set_error("the one-tile head GEMM needs vocab_size == 256"); return EGG_E_INVALID; }
    if (epi == EPI_LOGITS && p.N % 256) { set_error("the logits GEMM needs a vocabulary that is a multiple of 256"); return EGG_E_INVALID; }
    if (epi <= EPI_LOGITS) {
        int max_slots = ((GEMM_BM - 1) / p.seq_len) / 2 + 2;
        const bool rpl = p.seq_len % 32 == 0 && p.rpl >= 0;
        if (!rpl && max_slots > GEMM_MAX_SLOTS) { set_error("seq_len %d too small for the epilogue tables", p.seq_len); return EGG_E_INVALID; }
    }
    if (epi == EPI_VOTE && p.k_splits > 1) {
        // every split must own at least one k-block: the kernel cuts ceil(num_kb / k_splits) blocks per split
        const int num_kb = (p.K + GEMM_BK - 1) / GEMM_BK;
        const int kb_per = (num_kb + p.k_splits - 1) / p.k_splits;
        if ((num_kb + kb_per - 1) / kb_per != p.k_splits) { set_error("k_splits %d leaves an empty split of %d k-blocks", p.k_splits, num_kb); return EGG_E_INVALID; }
    }
    p.fd_seq = make_fastdiv(p.seq_len);
    p.fd_tiles_n = make_fastdiv(p.N / bn);
    p.fd_third = make_fastdiv(p.third);
    p.fd_head = make_fastdiv(p.head_dim);
    p.lut_stride = 32 * 4;
    p.one = 1;
    if (epi == EPI_GELU && p.out_shift + p.rank1_shift > PRESHIFT_MAX) {
        set_error("shifts %d + %d too large for the pre-shifted bias table", p.out_shift, p.rank1_shift);
        return EGG_E_INVALID;
    }
    p.pow_t = epi == EPI_GELU || epi == EPI_LOGITS ? merged_shift(p.K, p.rank1_shift, p.out_shift) : 0;
    CUtensorMap ta, tb;
    int rc;
    const int rows_m = (p.M + GEMM_BM - 1) / GEMM_BM;
    const bool pair = bn == 256 && pairs_form(epi, p, rows_m, num_sms);
    if ((rc = make_tmap(&ta, A, (uint64_t)p.M, (uint64_t)p.K, GEMM_BM))) return rc;
    if ((rc = make_tmap(&tb, B, (uint64_t)p.N, (uint64_t)p.K, (uint32_t)(pair ? bn / 2 : bn)))) return rc;
    CUtensorMap to = ta;       // only the row-per-lane int32 epilogues store through a tensor map
    if ((epi == EPI_PRE32 || epi == EPI_QKV) && p.seq_len % 32 == 0 && p.rpl >= 0) {
        if ((rc = make_tmap_out(&to, p.out32, (uint64_t)p.M, (uint64_t)p.N))) return rc;
    }
    if (epi == EPI_LOGITS || ((epi == EPI_GELU || epi == EPI_CLIP8) && bn == 256 && p.seq_len % 32 == 0 && p.rpl >= 0)) {
        if ((rc = make_tmap_out8(&to, p.out8, (uint64_t)p.M, (uint64_t)p.N))) return rc;
    }
    if (pair) {
        if (epi == EPI_VOTE) return launch_pair<EPI_VOTE, 0>(st, ta, tb, to, p, num_sms);
        return epi == EPI_GELU ? launch_pair<EPI_GELU, 1>(st, ta, tb, to, p, num_sms) : launch_pair<EPI_CLIP8, 1>(st, ta, tb, to, p, num_sms);
    }
    switch (epi) {
        case EPI_CLIP8: return launch_eval<EPI_CLIP8>(st, bn, ta, tb, to, p, num_sms);
        case EPI_GELU: return launch_eval<EPI_GELU>(st, bn, ta, tb, to, p, num_sms);
        case EPI_PRE32: return launch_eval<EPI_PRE32>(st, bn, ta, tb, to, p, num_sms);
        case EPI_QKV: return launch_eval<EPI_QKV>(st, bn, ta, tb, to, p, num_sms);
        case EPI_HEAD:
            if (p.seq_len % 32 == 0 && p.rpl >= 0) return launch_one<256, EPI_HEAD, 1>(st, ta, tb, to, p, num_sms);
            return launch_one<256, EPI_HEAD>(st, ta, tb, to, p, num_sms);
        case EPI_LOGITS:
            if (p.seq_len % 32 == 0 && p.rpl >= 0) return launch_one<256, EPI_LOGITS, 1>(st, ta, tb, to, p, num_sms);
            return launch_one<256, EPI_LOGITS>(st, ta, tb, to, p, num_sms);
        case EPI_VOTE: return launch_bn<EPI_VOTE>(st, bn, ta, tb, to, p, num_sms);
        case EPI_NULL: return launch_one<256, EPI_NULL>(st, ta, tb, to, p, num_sms);
    }
    set_error("unknown epilogue %d", epi);
    return EGG_E_INVALID;
}

}  // namespace egg
