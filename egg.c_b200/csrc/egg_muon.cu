// Muon (muon_internal.cuh:15-342): momentum, Frobenius normalise, five cubic Newton-Schulz steps
//     G = 3 I - X X^T  (or X^T X, whichever is smaller),   X <- 0.5 G X  (or 0.5 X G),
// and the quantised apply, for batches of equally shaped matrices.
//
// The products are fp32 products on the bf16 tensor cores.  A float is exactly the sum of three bf16 terms (8 + 8 + 8
// significant bits), and a product keeps the six of the nine partial products that reach 2^-24 of it:
//     hi*hi | hi*mid + mid*hi + mid*mid + hi*lo + lo*hi.
// hi*hi accumulates apart from the rest, and both leave tensor memory after every 64 contraction steps to be added to fp32
// registers with round-to-nearest: the tensor core's own additions truncate, and a chain of 4 is short enough not to show.
// Against fp64 the result is closer than the ordered chain of fused multiply-adds it replaces (tests/test_muon_gpu.py).
// Bound: tensor cores, six bf16 products per fp32 product; the Gram matrix is symmetric and computed once (by pairs of blocks: its diagonal
// tile pairs with one below the diagonal, which is formed and dropped).
#include "egg_muon.cuh"
#include "egg_ptx.cuh"

#include <cuda.h>

#include <algorithm>

namespace egg {

constexpr int NS_T = 128;                          // tile edge
constexpr int NS_K = 64;                           // contraction per stage: one 128-byte swizzled row of bf16
constexpr int NS_EPI_WARPS = 8;
constexpr int NS_THREADS = 64 + NS_EPI_WARPS * 32;
constexpr int NS_BOX = NS_T * NS_K * 2;

// CG == 2: pairs of blocks (cta_group::2) form two row tiles of the same columns, each with its own 128 rows of A and half of B's.
template <int CG>
struct NsSmem {
    static constexpr int ST = CG == 2 ? 3 : 2;         // stages
    alignas(1024) uint8_t a[ST][3][NS_BOX];
    alignas(1024) uint8_t b[ST][3][NS_BOX / CG];
    alignas(8) uint64_t full[ST], empty[ST], tmem_full[2], tmem_empty[2];
    uint32_t tmem_base;
    volatile int abort_flag;
};

enum { NS_GRAM = 0, NS_STEP = 1, NS_LAST = 2 };

struct NsParams {
    int nb, rows_a, rows_b, kdim;                  // per matrix: rows of A and of B, contraction length
    int tiles_i, tiles_j, tiles;                   // tiles of one matrix (GRAM: upper triangle)
    __nv_bfloat16 *out, *out_t;                    // three terms, [3][nb][rows_a][rows_b] and transposed (GRAM: out only)
    float *y;
    int *err;
};

__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_bf16_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// v = t[0] + t[1] + t[2] exactly (while the last term is above the smallest bf16)
__device__ __forceinline__ void split3(float v, __nv_bfloat16 (&t)[3]) {
    t[0] = __float2bfloat16_rn(v);
    const float r1 = v - __bfloat162float(t[0]);
    t[1] = __float2bfloat16_rn(r1);
    t[2] = __float2bfloat16_rn(r1 - __bfloat162float(t[1]));
}

template <int MODE, int CG>
__global__ void __launch_bounds__(NS_THREADS, 1)
ns_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const NsParams p) {
    extern __shared__ uint8_t ns_raw[];
    using Smem = NsSmem<CG>;
    constexpr int ST = Smem::ST;
    Smem &sm = *reinterpret_cast<Smem *>((reinterpret_cast<uintptr_t>(ns_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int items = p.tiles * p.nb, chunks = p.kdim / NS_K;
    const int prow = CG == 2 ? (int)(blockIdx.x & 1) : 0;           // this block's row tile of the pair (clusters are consecutive blocks)
    const int first_item = (int)blockIdx.x / CG, item_step = (int)gridDim.x / CG;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) { ptx::mbar_init(&sm.full[s], 1); ptx::mbar_init(&sm.empty[s], 1); }
        for (int a = 0; a < 2; a++) { ptx::mbar_init(&sm.tmem_full[a], 1); ptx::mbar_init(&sm.tmem_empty[a], CG * NS_EPI_WARPS); }
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
    if (CG == 2) ptx::cluster_sync_all();          // the other block's barriers exist before anything arrives on them
    const uint32_t tmem_base = sm.tmem_base;
    auto decode = [&](int item, int &mat, int &ti, int &tj) {
        mat = item / p.tiles;
        int t = item - mat * p.tiles;
        if (MODE == NS_GRAM) {                     // row ti of the upper triangle holds tiles_j - ti tiles, and so do the CG rows from it on
            ti = 0;
            while (t >= p.tiles_j - ti) { t -= p.tiles_j - ti; ti += CG; }
            tj = ti + t;
        } else {
            ti = t / p.tiles_j;
            tj = t - ti * p.tiles_j;
            ti *= CG;
        }
        ti += prow;
    };
    auto fail = [&](int code) {
        sm.abort_flag = 1;
        if (p.err) atomicCAS(p.err, 0, code);
    };
    if (warp == 0) {
        if (ptx::elect_one()) {
            uint32_t it = 0;
            bool ok = true;
            const uint32_t full_s = CG == 2 ? ptx::mapa_u32(ptx::smem_u32(sm.full), 0u) : 0u;          // of the even block
            for (int item = first_item; item < items && ok; item += item_step) {
                int mat, ti, tj;
                decode(item, mat, ti, tj);
                for (int c = 0; c < chunks; c++, it++) {
                    const int s = it % ST;
                    if (!ptx::mbar_wait(&sm.empty[s], ((it / ST) & 1) ^ 1) || sm.abort_flag) { fail(DEV_TIMEOUT_EMPTY); ok = false; break; }
                    if (prow == 0) ptx::mbar_arrive_expect_tx(&sm.full[s], 3 * CG * (NS_BOX + NS_BOX / CG));          // of both blocks
#pragma unroll
                    for (int q = 0; q < 3; q++) {
                        const int ya = (q * p.nb + mat) * p.rows_a + ti * NS_T, yb = (q * p.nb + mat) * p.rows_b + tj * NS_T + prow * (NS_T / CG);
                        if (CG == 2) {
                            ptx::tma_load_2d_pair(sm.a[s][q], &map_a, full_s + 8 * s, c * NS_K, ya);
                            ptx::tma_load_2d_pair(sm.b[s][q], &map_b, full_s + 8 * s, c * NS_K, yb);
                        } else {
                            ptx::tma_load_2d(sm.a[s][q], &map_a, &sm.full[s], c * NS_K, ya);
                            ptx::tma_load_2d(sm.b[s][q], &map_b, &sm.full[s], c * NS_K, yb);
                        }
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
            // bf16 x bf16 -> fp32, both operands K-major, 128 columns
            constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NS_T >> 3) << 17) | ((uint32_t)(CG * NS_T >> 4) << 24);
            uint32_t it = 0;
            bool ok = true;
            for (int item = first_item; item < items && ok; item += item_step) {
                for (int c = 0; c < chunks; c++, it++) {
                    const int s = it % ST, as = it & 1;
                    if (!ptx::mbar_wait(&sm.tmem_empty[as], ((it >> 1) & 1) ^ 1) || sm.abort_flag) { fail(DEV_TIMEOUT_TMEM_EMPTY); ok = false; break; }
                    if (!ptx::mbar_wait(&sm.full[s], (it / ST) & 1) || sm.abort_flag) { fail(DEV_TIMEOUT_FULL); ok = false; break; }
                    ptx::tc_fence_after();
                    const uint32_t d0 = tmem_base + (uint32_t)(as * 2 * NS_T), d1 = d0 + NS_T;
                    uint64_t a[3], b[3];
#pragma unroll
                    for (int q = 0; q < 3; q++) {
                        a[q] = ptx::make_smem_desc_sw128(ptx::smem_u32(sm.a[s][q]));
                        b[q] = ptx::make_smem_desc_sw128(ptx::smem_u32(sm.b[s][q]));
                    }
#pragma unroll
                    for (int k = 0; k < NS_K / 16; k++) {
                        const uint64_t o = (uint64_t)(2 * k);          // 16 bf16 = 32 bytes along the swizzled row
                        auto mma = [&](uint32_t d, int i, int j, uint32_t more) {
                            if (CG == 2) mma_bf16_pair(d, a[i] + o, b[j] + o, idesc, more); else mma_bf16(d, a[i] + o, b[j] + o, idesc, more);
                        };
                        mma(d1, 0, 2, k > 0);
                        mma(d1, 2, 0, 1);
                        mma(d1, 1, 1, 1);
                        mma(d1, 0, 1, 1);
                        mma(d1, 1, 0, 1);
                        mma(d0, 0, 0, k > 0);
                    }
                    if (CG == 2) { ptx::mma_commit_pair(&sm.empty[s], 0); ptx::mma_commit_pair(&sm.tmem_full[as], 0); }
                    else { ptx::mma_commit(&sm.empty[s]); ptx::mma_commit(&sm.tmem_full[as]); }
                }
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const uint32_t tmem_empty_s = CG == 2 ? ptx::mapa_u32(ptx::smem_u32(sm.tmem_empty), 0u) : 0u;          // of the even block
        uint32_t it = 0;
        bool ok = true;
        for (int item = first_item; item < items && ok; item += item_step) {
            int mat, ti, tj;
            decode(item, mat, ti, tj);
            float acc[64];
#pragma unroll
            for (int i = 0; i < 64; i++) acc[i] = 0.0f;
            for (int c = 0; c < chunks; c++, it++) {
                const int as = it & 1;
                ok = ptx::mbar_wait(&sm.tmem_full[as], (it >> 1) & 1) && !sm.abort_flag;
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (!ok) { if (lane == 0) fail(DEV_TIMEOUT_TMEM_FULL); break; }
                ptx::tc_fence_after();
                const uint32_t ta = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(as * 2 * NS_T + half * 64);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    uint32_t u[16], v[16];
                    ptx::tmem_ld16(ta + 16 * q, u);
                    ptx::tmem_ld16(ta + NS_T + 16 * q, v);
                    ptx::tmem_ld_wait16(u);
                    ptx::tmem_ld_wait16(v);
#pragma unroll
                    for (int i = 0; i < 16; i++) acc[16 * q + i] += __uint_as_float(u[i]) + __uint_as_float(v[i]);
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (CG == 2) ptx::mbar_arrive_peer(tmem_empty_s + 8 * as); else ptx::mbar_arrive(&sm.tmem_empty[as]);
                }
            }
            if (!ok) break;
            if (MODE == NS_GRAM && CG == 2 && ti > tj) continue;            // below the diagonal: the pair's other tile is the diagonal one
            const int i = ti * NS_T + quarter * 32 + lane, j0 = tj * NS_T + half * 64;
            if (MODE == NS_LAST) {
                float *o = p.y + ((int64_t)mat * p.rows_a + i) * p.rows_b + j0;
#pragma unroll
                for (int q = 0; q < 16; q++) *reinterpret_cast<float4 *>(o + 4 * q) = make_float4(0.5f * acc[4 * q], 0.5f * acc[4 * q + 1], 0.5f * acc[4 * q + 2], 0.5f * acc[4 * q + 3]);
            } else {
                const int64_t term = (int64_t)p.nb * p.rows_a * p.rows_b;
                __nv_bfloat16 *o = p.out + ((int64_t)mat * p.rows_a + i) * p.rows_b + j0;
                // transposed: [rows_b][rows_a]; the Gram matrix mirrors its upper triangle into itself
                __nv_bfloat16 *ot = (MODE == NS_GRAM ? p.out : p.out_t) + ((int64_t)mat * p.rows_b + j0) * p.rows_a + i;
                const bool mirror = MODE == NS_STEP || ti != tj;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    union { __nv_bfloat16 h[8]; uint4 v; } w[3];
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int j = 8 * q + k;
                        float v = MODE == NS_GRAM ? -acc[j] : 0.5f * acc[j];
                        if (MODE == NS_GRAM && i == j0 + j) v = 3.0f - acc[j];         // muon_newton_schulz_term_kernel, muon_internal.cuh:91-109
                        __nv_bfloat16 t[3];
                        split3(v, t);
#pragma unroll
                        for (int s = 0; s < 3; s++) {
                            w[s].h[k] = t[s];
                            if (mirror) ot[s * term + (int64_t)j * p.rows_a] = t[s];
                        }
                    }
#pragma unroll
                    for (int s = 0; s < 3; s++) *reinterpret_cast<uint4 *>(o + s * term + 8 * q) = w[s].v;
                }
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

template <int MODE>
static int ns_init() {
    EGG_CUDA(cudaFuncSetAttribute(ns_gemm_kernel<MODE, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(NsSmem<1>) + 1024));
    EGG_CUDA(cudaFuncSetAttribute(ns_gemm_kernel<MODE, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(NsSmem<2>) + 1024));
    return EGG_OK;
}

int muon_init() {
    static bool done[EGG_MAX_DEVICES] = {};
    bool &d = done[current_device_slot()];
    if (d) return EGG_OK;
    int rc;
    if ((rc = ns_init<NS_GRAM>()) || (rc = ns_init<NS_STEP>()) || (rc = ns_init<NS_LAST>())) return rc;
    d = true;
    return EGG_OK;
}

int64_t ns_ws_bytes(int rows, int cols, int nb) {
    const int64_t n = (int64_t)rows * cols, k = rows < cols ? rows : cols;
    return nb * (n * (4 * 6 + 4) + k * k * 6) + 4096;
}
void ns_ws_carve(NsWs &ws, void *base, int rows, int cols, int nb) {
    const int64_t n = (int64_t)nb * rows * cols, k = rows < cols ? rows : cols;
    uint8_t *b = static_cast<uint8_t *>(base);
    auto take = [&](int64_t bytes) { void *q = b; b += (bytes + 255) & ~(int64_t)255; return q; };
    for (int i = 0; i < 2; i++) {
        ws.xr[i] = static_cast<__nv_bfloat16 *>(take(n * 6));
        ws.xc[i] = static_cast<__nv_bfloat16 *>(take(n * 6));
    }
    ws.g = static_cast<__nv_bfloat16 *>(take((int64_t)nb * k * k * 6));
    ws.y = static_cast<float *>(take(n * 4));
}

template <int MODE>
static int launch_ns_gemm(cudaStream_t st, const __nv_bfloat16 *a, const __nv_bfloat16 *b, NsParams p, int num_sms) {
    CUtensorMap ma, mb;
    int rc;
    p.tiles_i = p.rows_a / NS_T; p.tiles_j = p.rows_b / NS_T;
    // Pairs from a smaller side of 512 on, where row tiles come in pairs.  A 128 x 128 tile in six products reads 128 bytes a clock from shared
    // memory and 64 from L2 at the tensor cores' rate, a pair's 96 and 48.  Five steps of one 4096 x 4096 matrix 5.1 -> 4.5 ms, of the
    // matrices of four layers at H 1024 17.9 -> 16.6, at H 768 (two layers) 4.38 -> 4.22; at H 512 a whole update 1.44 -> 1.43, at H 256 0.440 -> 0.444.
    const int cg = std::min(p.rows_a, std::min(p.rows_b, p.kdim)) >= 512 && p.tiles_i % 2 == 0 ? 2 : 1;
    if ((rc = bf16_tensor_map(&ma, a, 3ull * p.nb * p.rows_a, (uint64_t)p.kdim, NS_T)) || (rc = bf16_tensor_map(&mb, b, 3ull * p.nb * p.rows_b, (uint64_t)p.kdim, NS_T / cg))) return rc;
    if (cg == 1) {
        p.tiles = MODE == NS_GRAM ? p.tiles_i * (p.tiles_i + 1) / 2 : p.tiles_i * p.tiles_j;
        const int items = p.tiles * p.nb;
        ns_gemm_kernel<MODE, 1><<<items < num_sms ? items : num_sms, NS_THREADS, sizeof(NsSmem<1>) + 1024, st>>>(ma, mb, p);
        EGG_CUDA(cudaGetLastError());
        return EGG_OK;
    }
    p.tiles = MODE == NS_GRAM ? p.tiles_i / 2 * (p.tiles_i / 2 + 1) : p.tiles_i / 2 * p.tiles_j;          // pairs of tiles
    const int items = p.tiles * p.nb;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(NS_THREADS); cfg.dynamicSmemBytes = sizeof(NsSmem<2>) + 1024; cfg.stream = st; cfg.attrs = attr; cfg.numAttrs = 1;
    cfg.gridDim = dim3((unsigned)(2 * (items < num_sms / 2 ? items : num_sms / 2)));
    EGG_CUDA(cudaLaunchKernelEx(&cfg, ns_gemm_kernel<MODE, 2>, ma, mb, p));
    return EGG_OK;
}

int launch_newton_schulz(cudaStream_t st, const NsWs &ws, int rows, int cols, int nb, int *err, int num_sms) {
    if (rows % NS_T || cols % NS_T || nb < 1) { set_error("Newton-Schulz shape %d x %d unsupported", rows, cols); return EGG_E_INVALID; }
    const bool use_rows = rows < cols;
    const int K = use_rows ? rows : cols;
    int cur = 0, rc;
    for (int it = 0; it < 5; it++, cur ^= 1) {
        NsParams g = {};
        g.nb = nb; g.rows_a = g.rows_b = K; g.kdim = use_rows ? cols : rows; g.out = ws.g; g.err = err;
        const __nv_bfloat16 *x = use_rows ? ws.xr[cur] : ws.xc[cur];
        if ((rc = launch_ns_gemm<NS_GRAM>(st, x, x, g, num_sms))) return rc;
        NsParams s = {};
        s.nb = nb; s.rows_a = rows; s.rows_b = cols; s.kdim = K; s.out = ws.xr[cur ^ 1]; s.out_t = ws.xc[cur ^ 1]; s.y = ws.y; s.err = err;
        const __nv_bfloat16 *a = use_rows ? ws.g : ws.xr[cur], *b = use_rows ? ws.xc[cur] : ws.g;
        if ((rc = it < 4 ? launch_ns_gemm<NS_STEP>(st, a, b, s, num_sms) : launch_ns_gemm<NS_LAST>(st, a, b, s, num_sms))) return rc;
    }
    return EGG_OK;
}

// ------------------------------------------------------------------ element passes; a block owns 32 outputs n x 128 inputs k
__global__ void __launch_bounds__(256) muon_momentum_kernel(const UpdMat *mats, const int *list, const int32_t *votes, int splits, int64_t split_stride,
                                                            uint8_t *opt, float mu, double *norm2) {
    __shared__ double part[8];
    const UpdMat &m = mats[list[blockIdx.y]];
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5, bn = m.cols_n / 32;
    const int n = ((int)blockIdx.x % bn) * 32 + lane, kq0 = ((int)blockIdx.x / bn) * 32;
    double ss = 0;                                 // the norm feeds one fp32 division per element
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int64_t word = (int64_t)(kq0 + ty + 8 * i) * m.cols_n + n;
        int4 vt = *reinterpret_cast<const int4 *>(votes + m.votes_off + word * 4);
        for (int s = 1; s < splits; s++) {
            const int4 u = *reinterpret_cast<const int4 *>(votes + (int64_t)s * split_stride + m.votes_off + word * 4);
            vt.x += u.x; vt.y += u.y; vt.z += u.z; vt.w += u.w;
        }
        float4 *sp = reinterpret_cast<float4 *>(opt + m.opt_off) + word * 2;          // {m, acc} pairs
        float4 s0 = sp[0], s1 = sp[1];
        s0.x = __fmaf_rn(mu, s0.x, (float)vt.x);   // m = mu*m + vote, muon_internal.cuh:45-47
        s0.z = __fmaf_rn(mu, s0.z, (float)vt.y);
        s1.x = __fmaf_rn(mu, s1.x, (float)vt.z);
        s1.z = __fmaf_rn(mu, s1.z, (float)vt.w);
        sp[0] = s0; sp[1] = s1;
        ss += (double)s0.x * s0.x + (double)s0.z * s0.z + (double)s1.x * s1.x + (double)s1.z * s1.z;
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
    if (lane == 0) part[ty] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int i = 0; i < 8; i++) t += part[i];
        atomicAdd(&norm2[blockIdx.y], t);
    }
}
int launch_muon_momentum(cudaStream_t st, const UpdMat *mats, const int *list, int nb, int rows, int cols, const int32_t *votes, int splits,
                         int64_t split_stride, uint8_t *opt, float mu, double *norm2) {
    muon_momentum_kernel<<<dim3((unsigned)(cols / 32 * (rows / 128)), (unsigned)nb), 256, 0, st>>>(mats, list, votes, splits, split_stride, opt, mu, norm2);
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

__global__ void __launch_bounds__(256) muon_split_kernel(const UpdMat *mats, const int *list, int nb, const uint8_t *opt, const double *norm2, __nv_bfloat16 *xr,
                                                         __nv_bfloat16 *xc) {
    __shared__ float tile[128][33];
    const UpdMat &m = mats[list[blockIdx.y]];
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5, bn = m.cols_n / 32, R = m.rows_k, C = m.cols_n;
    const int n0 = ((int)blockIdx.x % bn) * 32, k0 = ((int)blockIdx.x / bn) * 128;
    const float norm = (float)sqrt(norm2[blockIdx.y]);
    const bool div = norm > 1e-6f;                 // muon_scale_by_norm_kernel, muon_internal.cuh:77-85
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int kq = ty + 8 * i;
        const float4 *sp = reinterpret_cast<const float4 *>(opt + m.opt_off) + ((int64_t)(k0 / 4 + kq) * C + n0 + lane) * 2;
        const float4 s0 = sp[0], s1 = sp[1];
        const float v[4] = {s0.x, s0.z, s1.x, s1.z};
#pragma unroll
        for (int j = 0; j < 4; j++) tile[4 * kq + j][lane] = div ? __fdiv_rn(v[j], norm) : v[j];
    }
    __syncthreads();
    const int64_t term = (int64_t)nb * R * C;
    for (int e = threadIdx.x; e < 128 * 16; e += 256) {          // row-major: two outputs n per thread
        const int k = e >> 4, n = (e & 15) * 2;
        __nv_bfloat16 a[3], b[3];
        split3(tile[k][n], a);
        split3(tile[k][n + 1], b);
        __nv_bfloat16 *o = xr + ((int64_t)blockIdx.y * R + k0 + k) * C + n0 + n;
#pragma unroll
        for (int s = 0; s < 3; s++) *reinterpret_cast<__nv_bfloat162 *>(o + s * term) = __nv_bfloat162(a[s], b[s]);
    }
    for (int e = threadIdx.x; e < 32 * 64; e += 256) {           // transposed: two inputs k per thread
        const int n = e >> 6, k = (e & 63) * 2;
        __nv_bfloat16 a[3], b[3];
        split3(tile[k][n], a);
        split3(tile[k + 1][n], b);
        __nv_bfloat16 *o = xc + ((int64_t)blockIdx.y * C + n0 + n) * R + k0 + k;
#pragma unroll
        for (int s = 0; s < 3; s++) *reinterpret_cast<__nv_bfloat162 *>(o + s * term) = __nv_bfloat162(a[s], b[s]);
    }
}
int launch_muon_split(cudaStream_t st, const UpdMat *mats, const int *list, int nb, int rows, int cols, const uint8_t *opt, const double *norm2, const NsWs &ws) {
    muon_split_kernel<<<dim3((unsigned)(cols / 32 * (rows / 128)), (unsigned)nb), 256, 0, st>>>(mats, list, nb, opt, norm2, ws.xr[0], ws.xc[0]);
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

// muon_apply_update_kernel (muon_internal.cuh:112-166); the new weights also leave in the K-major copy
__global__ void __launch_bounds__(256) muon_apply_kernel(const UpdMat *mats, const int *list, const float *y, int8_t *model, uint8_t *opt, int8_t *shadow,
                                                         float lr0, float wd, unsigned long long *total) {
    __shared__ uint32_t tile[32][33];
    __shared__ int s_changes;
    const UpdMat &m = mats[list[blockIdx.y]];
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5, bn = m.cols_n / 32, C = m.cols_n;
    const int n0 = ((int)blockIdx.x % bn) * 32, kq0 = ((int)blockIdx.x / bn) * 32;
    const float lr = lr0 * m.lr_scale;
    if (threadIdx.x == 0) s_changes = 0;
    __syncthreads();
    int changes = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int kq = kq0 + ty + 8 * i;
        const int64_t word = (int64_t)kq * C + n0 + lane;
        const float *u = y + ((int64_t)blockIdx.y * m.rows_k + 4 * kq) * C + n0 + lane;
        uint32_t *wp = reinterpret_cast<uint32_t *>(model + m.model_off) + word;
        float4 *sp = reinterpret_cast<float4 *>(opt + m.opt_off) + word * 2;
        float4 s0 = sp[0], s1 = sp[1];
        float acc[4] = {s0.y, s0.w, s1.y, s1.w};
        const uint32_t wword = *wp;
        uint32_t neww = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            int w = (int)(int8_t)(wword >> (8 * j));
            acc[j] = __fmaf_rn(-lr, __fmaf_rn(wd, (float)w, u[(int64_t)j * C]), acc[j]);     // acc += -lr*(u + wd*w), contracted as nvcc does
            changes += quantized_step(acc[j], w);
            neww |= (uint32_t)(w & 0xFF) << (8 * j);
        }
        s0.y = acc[0]; s0.w = acc[1]; s1.y = acc[2]; s1.w = acc[3];
        *wp = neww;
        sp[0] = s0; sp[1] = s1;
        tile[ty + 8 * i][lane] = neww;
    }
    changes = __reduce_add_sync(0xFFFFFFFFu, changes);
    if (lane == 0 && changes) atomicAdd(&s_changes, changes);
    __syncthreads();
    if (shadow) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int nn = ty + 8 * i;
            *reinterpret_cast<uint32_t *>(shadow + m.shadow_off + (int64_t)(n0 + nn) * m.rows_k + 4 * (kq0 + lane)) = tile[lane][nn];
        }
    }
    if (threadIdx.x == 0 && s_changes) atomicAdd(total, (unsigned long long)s_changes);
}
int launch_muon_apply(cudaStream_t st, const UpdMat *mats, const int *list, int nb, int rows, int cols, const float *y, int8_t *model, uint8_t *opt,
                      int8_t *shadow, float lr, float wd, unsigned long long *total) {
    muon_apply_kernel<<<dim3((unsigned)(cols / 32 * (rows / 128)), (unsigned)nb), 256, 0, st>>>(mats, list, y, model, opt, shadow, lr, wd, total);
    EGG_CUDA(cudaGetLastError());
    return EGG_OK;
}

}  // namespace egg
