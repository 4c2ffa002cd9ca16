// Sampling: one un-perturbed stream decoded token by token with a KV cache
// (generate_sequence_kernel, d-eggs/src/kernels.cu:307-490; mgpu.cu:1154-1285 is the case temp = 1,
// no min-p filter, no presence penalty).
//
// Serial over tokens and one row wide: the work of a token is to read every weight once and to pass a few hundred bytes
// from product to product.  One cluster of 16 blocks shares each product's outputs; its rows of the K-major weight copies
// are contiguous, so one warp per block streams them from L2 through a ring of bulk copies, running ahead of the data by
// up to 160 KB, while eight warps form the dot products.  Results go to all blocks as st.async stores counted by a
// transaction mbarrier in the receiver, and everything between two products (residual, adaptive normalise, mean-abs norm,
// RoPE, the draw) is repeated by every block, so that a product costs one exchange and no second trip.  Attention of head
// i runs in block i, whose threads hold their context's K row and V pieces in registers before the exchange completes.
// Bound: latency (5 layers + 3 exchanges per token) up to about 15 MB of weights, L2 to 16 SMs (64 B per clock each) above.
#include "egg_kernels.cuh"

#include <limits.h>

namespace egg {

constexpr int GEN_BLOCKS = 16;
constexpr int GEN_WARPS = 8;                       // compute warps; one more streams the weights
constexpr int GEN_CT = GEN_WARPS * 32;
constexpr int GEN_THREADS = GEN_CT + 32;
constexpr int GEN_STAGES = 5;
constexpr int GEN_CHUNK = 32768;

struct GenSmem {
    alignas(128) int8_t ring[GEN_STAGES][GEN_CHUNK];
    alignas(16) int32_t qkv[3 * 1024];             // exchanged: q | k | v before RoPE
    alignas(16) int32_t po[1024], pd[1024];        // exchanged: output and down products
    alignas(16) int32_t logits[256];               // exchanged
    alignas(16) int8_t u[4096], ao[1024];          // exchanged: MLP activations, attention output
    alignas(16) int8_t h[1024];                    // this block's copy of the normalised row
    alignas(16) int8_t q8[64], k8[64], v8[64];     // the new token's rows of this block's head
    alignas(16) long long part[GEN_WARPS][64];     // attention: Σ w·v of each warp's contexts
    int32_t wt[256];                               // attention weights; later the exp values of the draw
    alignas(16) int32_t red[8][GEN_WARPS];
    int32_t exp_lut[256];
    int32_t count[256];                            // occurrences of every token so far
    int8_t act_lut[256];
    uint8_t tok[256];
    int32_t sel;
    alignas(8) uint64_t full[GEN_STAGES], empty[GEN_STAGES], ex[2];
    volatile int dead;
};

struct GenState {                                  // per compute thread
    uint32_t ring_it;                              // ring chunks consumed so far
    uint32_t ex_it;                                // exchanges completed so far
    int rank, warp, lane, tid;
    uint32_t smem_base;
};

__device__ __forceinline__ bool gen_wait(GenSmem &s, uint64_t *bar, uint32_t parity, int *err) {
    for (int i = 0; i < (1 << 20); i++) {          // bounded: each try is suspended for up to 2 us
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred P;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, P;\n\t}"
            : "=r"(ok)
            : "r"(ptx::smem_u32(bar)), "r"(parity), "r"(2000u)
            : "memory");
        if (ok) return true;
        if (s.dead) return false;
    }
    s.dead = 1;
    if (err) atomicCAS(err, 0, (int)DEV_TIMEOUT_PEER);
    return false;
}
// a ring stage: filled and emptied within this block, and mostly ahead of its use
__device__ __forceinline__ void gen_wait_ring(GenSmem &s, uint64_t *bar, uint32_t parity, int *err) {
    if (!ptx::mbar_try_wait(bar, parity)) gen_wait(s, bar, parity, err);
}
__device__ __forceinline__ void gen_bar() { ptx::named_bar_sync(1, GEN_CT); }
__device__ __forceinline__ void st_async_b32(uint32_t addr, uint32_t bar, uint32_t v) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %2, [%1];" ::"r"(addr), "r"(bar), "r"(v) : "memory");
}
__device__ __forceinline__ void st_async_v2(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%2, %3}, [%1];" ::"r"(addr), "r"(bar), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, int a, int b, int c, int d) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(addr), "r"(bar), "r"(a), "r"(b),
                 "r"(c), "r"(d)
                 : "memory");
}

// rows of one ring chunk: as many as fit, in whole groups of `group`
__host__ __device__ __forceinline__ int gen_chunk_rows(int K, int left, int group) {
    const int fit = GEN_CHUNK / K / group * group;
    return left < fit ? left : fit;
}

// ---- producer: this block's rows of one matrix (K-major, rank's share contiguous) into the ring ----
__device__ __forceinline__ void gen_stream(GenSmem &s, uint32_t &it, const int8_t *w, int rank, int rows, int K, int group, int *err) {
    const int8_t *src = w + (int64_t)rank * rows * K;
    for (int r = 0; r < rows;) {
        const int rc = gen_chunk_rows(K, rows - r, group);
        const int st = it % GEN_STAGES;
        if (s.dead || !gen_wait(s, &s.empty[st], ((it / GEN_STAGES) & 1) ^ 1, err)) return;
        ptx::mbar_arrive_expect_tx(&s.full[st], (uint32_t)(rc * K));
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(ptx::smem_u32(s.ring[st])),
                     "l"(src + (int64_t)r * K), "r"(rc * K), "r"(ptx::smem_u32(&s.full[st]))
                     : "memory");
        it++;
        r += rc;
    }
}

// ---- consumer: dot products of the block's rows with a vector kept in registers ----
// Lane l holds the vector's words in the order the row words are read: KW words as 16-, 8- or 4-byte pieces.
template <int KW>
__device__ __forceinline__ void gen_load_vec(const int8_t *v, int lane, int32_t (&x)[KW]) {
    constexpr int P = KW % 4 == 0 ? 4 : (KW % 2 == 0 ? 2 : 1);
#pragma unroll
    for (int j = 0; j < KW / P; j++)
#pragma unroll
        for (int i = 0; i < P; i++) x[j * P + i] = *reinterpret_cast<const int32_t *>(v + (j * 32 + lane) * 4 * P + 4 * i);
}
template <int KW>
__device__ __forceinline__ int gen_dot(const int8_t *row, int lane, const int32_t (&x)[KW]) {
    constexpr int P = KW % 4 == 0 ? 4 : (KW % 2 == 0 ? 2 : 1);
    int a = 0;
#pragma unroll
    for (int j = 0; j < KW / P; j++) {
        const int8_t *p = row + (j * 32 + lane) * 4 * P;
        if (P == 4) {
            const int4 w = *reinterpret_cast<const int4 *>(p);
            a = __dp4a(w.x, x[j * P], a); a = __dp4a(w.y, x[j * P + 1], a); a = __dp4a(w.z, x[j * P + 2], a); a = __dp4a(w.w, x[j * P + 3], a);
        } else if (P == 2) {
            const int2 w = *reinterpret_cast<const int2 *>(p);
            a = __dp4a(w.x, x[j * P], a); a = __dp4a(w.y, x[j * P + 1], a);
        } else {
            a = __dp4a(*reinterpret_cast<const int32_t *>(p), x[j], a);
        }
    }
    return a;
}

// Sums of R rows over the warp, in every lane.
template <int KW, int R>
__device__ __forceinline__ void gen_rows(const int8_t *w, int lane, const int32_t (&x)[KW], int (&a)[R]) {
#pragma unroll
    for (int k = 0; k < R; k++) a[k] = gen_dot<KW>(w + k * KW * 128, lane, x);
#pragma unroll
    for (int k = 0; k < R; k++) a[k] = __reduce_add_sync(0xFFFFFFFFu, a[k]);
}
// The byte GELU[clip((sum >> shift) + bias)] of row lane & 3, and four bytes to a word: one look-up a lane, not four in a row.
__device__ __forceinline__ uint32_t gen_gelu4(GenSmem &s, int lane, const int (&a)[4], int bl, int i, int shift) {
    const int v = lane & 2 ? (lane & 1 ? a[3] : a[2]) : (lane & 1 ? a[1] : a[0]);
    const int b = __shfl_sync(0xFFFFFFFFu, bl, i + (lane & 3));
    const uint32_t byte = (uint32_t)(uint8_t)s.act_lut[(uint8_t)(int8_t)clip8((v >> shift) + b)] << (8 * (lane & 3));
    return __reduce_or_sync(0xFFFFFFFFu, lane < 4 ? byte : 0u);
}
// Eight rows with four lanes to a row: the sums meet in two shuffles, where a row a warp needs a warp-wide sum each (16 cycles of its
// unit with eight warps).  The quads read 64 bytes of their rows at a time, in odd rows the other half of 128 first, so that eight
// lanes cover all banks; x holds the vector's words in that order.
template <int NJ>
__device__ __forceinline__ void gen_load_quad(const int8_t *v, int lane, int4 (&x)[2 * NJ]) {
#pragma unroll
    for (int c = 0; c < 2 * NJ; c++) x[c] = *reinterpret_cast<const int4 *>(v + 64 * (c ^ (lane >> 2 & 1)) + 16 * (lane & 3));
}
template <int NJ>
__device__ __forceinline__ int gen_quad_dot(const int8_t *w, int lane, const int4 (&x)[2 * NJ]) {
    const int8_t *p = w + (lane >> 2) * (128 * NJ) + 16 * (lane & 3);
    int a = 0, b = 0;                         // two chains
#pragma unroll
    for (int c = 0; c < 2 * NJ; c++) {
        const int4 r = *reinterpret_cast<const int4 *>(p + 64 * (c ^ (lane >> 2 & 1)));
        int &t = c & 1 ? b : a;
        t = __dp4a(r.x, x[c].x, t); t = __dp4a(r.y, x[c].y, t); t = __dp4a(r.z, x[c].z, t); t = __dp4a(r.w, x[c].w, t);
    }
    return a + b;
}
// Their bytes GELU[clip((sum >> shift) + bias)] as two words, bl the bias of row lane / 4 (in every lane; the words are right in lanes 0-15).
__device__ __forceinline__ void gen_quad_gelu(GenSmem &s, int lane, int a, int bl, int shift, uint32_t (&word)[2]) {
    a += __shfl_xor_sync(0xFFFFFFFFu, a, 1);
    a += __shfl_xor_sync(0xFFFFFFFFu, a, 2);
    uint32_t w = (uint32_t)(uint8_t)s.act_lut[(uint8_t)(int8_t)clip8((a >> shift) + bl)] << (8 * (lane >> 2 & 3));
    w |= __shfl_xor_sync(0xFFFFFFFFu, w, 4);
    w |= __shfl_xor_sync(0xFFFFFFFFu, w, 8);
    word[0] = w;
    word[1] = __shfl_xor_sync(0xFFFFFFFFu, w, 16);
}

// out_off: byte offset of the product's exchange buffer inside GenSmem.  Every warp takes rc / 8 consecutive rows of a chunk.  How many
// run side by side is what a token's time hangs on (chains of loads, products, sums and a message): four rows where there are as many,
// eight of the up product at H 256, 384 and 512 by quads of lanes, those of two chunks at H 512; one or two rows of each of two
// neighbouring chunks, as in the down product, together.  What no chunk of a product can hold is not compiled: the instructions of a
// token are fetched anew for every product.  Against one row or four after another (256 bytes sampled, 2 layers): H 256 4.48 -> 3.88 ms,
// 384 4.86 -> 4.59, 640 6.45 -> 6.12, 768 7.50 -> 7.30, 1024 8.84 -> 8.41; 4 layers, H 512 7.82 -> 7.27.
// BYTES = false: int32 results; true: GELU[clip((acc >> shift) + bias)].
template <int KW, bool BYTES>
__device__ __forceinline__ void gen_product(GenSmem &s, GenState &g, const int8_t *vec, int rows, int group, uint32_t out_off, uint32_t bar_off, int *err,
                                            const int8_t *bias = nullptr, int shift = 0) {
    constexpr int K = KW * 128;
    constexpr bool QUADS = BYTES && KW >= 2 && KW <= 4;      // chunks of 64 rows and more
    constexpr int MOST = GEN_CHUNK / K / GEN_WARPS;          // most rows of a warp and chunk
    constexpr bool CHUNK_PAIRS = KW != 24;                   // (H 768: 7.46 ms with them, 7.35 without)
    const int dest = g.lane & 15, half = g.lane >> 4;
    const uint32_t bar = ptx::mapa_u32(g.smem_base + bar_off, dest);
    auto stage = [&](uint32_t k) { return (int)((g.ring_it + k) % GEN_STAGES); };
    auto wait_full = [&](uint32_t k) {
        const uint32_t it = g.ring_it + k;
        gen_wait_ring(s, &s.full[it % GEN_STAGES], (it / GEN_STAGES) & 1, err);
    };
    int r = 0;
    if constexpr (QUADS) {
        int4 x[2 * KW];
        gen_load_quad<KW>(vec, g.lane, x);
        constexpr int RC = 32768 / K / 32 * 32 < 32 * KW ? 32768 / K / 32 * 32 : 32 * KW, N = 32 * KW / RC;        // rows of a chunk, whole chunks
        static_assert(RC == 64 && GEN_CHUNK == 32768, "eight rows a warp and chunk");
        const int row0 = g.rank * rows + 8 * g.warp;
        int bl[N], a[N];
#pragma unroll
        for (int n = 0; n < N; n++) bl[n] = (int)bias[row0 + RC * n + (g.lane >> 2)];
#pragma unroll
        for (int n = 0; n < N; n++) {
            wait_full((uint32_t)n);
            __syncwarp();
            a[n] = gen_quad_dot<KW>(s.ring[stage((uint32_t)n)] + g.warp * 8 * K, g.lane, x);
        }
#pragma unroll
        for (int n = 0; n < N; n++) {
            uint32_t v[2];
            gen_quad_gelu(s, g.lane, a[n], bl[n], shift, v);
            if (half == 0) st_async_v2(ptx::mapa_u32(g.smem_base + out_off + row0 + RC * n, dest), bar, v[0], v[1]);
        }
        __syncwarp();
#pragma unroll
        for (int n = 0; n < N; n++)
            if (g.lane == 0) ptx::mbar_arrive(&s.empty[stage((uint32_t)n)]);
        g.ring_it += N;
        r = RC * N;
        if (KW != 3) return;
    }
    int32_t x[KW];
    gen_load_vec<KW>(vec, g.lane, x);
    while (r < rows) {
        const int rc = gen_chunk_rows(K, rows - r, group), per = rc / GEN_WARPS;
        const int st = stage(0);
        const int row0 = g.rank * rows + r + g.warp * per;            // row of the whole product
        const int bl = (BYTES && g.lane < per) ? (int)bias[row0 + g.lane] : 0;
        wait_full(0);
        if (!BYTES && MOST <= 2 && CHUNK_PAIRS && per <= 2 && rows - r >= 2 * rc) {
            // one or two rows of this chunk and as many of the next: lanes 0-15 send those, 16-31 these
            wait_full(1);
            __syncwarp();
            const int8_t *w0 = s.ring[st] + g.warp * per * K, *w1 = s.ring[stage(1)] + g.warp * per * K;
            const uint32_t at = ptx::mapa_u32(g.smem_base + out_off + 4 * (row0 + half * rc), dest);
            int a[4];
            a[0] = gen_dot<KW>(w0, g.lane, x); a[1] = gen_dot<KW>(w1, g.lane, x);
            if (per == 2) {
                a[2] = gen_dot<KW>(w0 + K, g.lane, x); a[3] = gen_dot<KW>(w1 + K, g.lane, x);
#pragma unroll
                for (int k = 0; k < 4; k++) a[k] = __reduce_add_sync(0xFFFFFFFFu, a[k]);
                st_async_v2(at, bar, (uint32_t)(half ? a[1] : a[0]), (uint32_t)(half ? a[3] : a[2]));
            } else {
#pragma unroll
                for (int k = 0; k < 2; k++) a[k] = __reduce_add_sync(0xFFFFFFFFu, a[k]);
                st_async_b32(at, bar, (uint32_t)(half ? a[1] : a[0]));
            }
            __syncwarp();
            if (g.lane == 0) { ptx::mbar_arrive(&s.empty[st]); ptx::mbar_arrive(&s.empty[stage(1)]); }
            g.ring_it += 2;
            r += 2 * rc;
            continue;
        }
        __syncwarp();
        const int8_t *w = s.ring[st] + (int64_t)g.warp * per * K;
        for (int i = 0; i < per;) {
            const uint32_t at = g.smem_base + out_off + (BYTES ? 1 : 4) * (row0 + i);
            if (MOST >= 4 && (BYTES || per - i >= 4)) {          // (the up product's chunks are whole groups of four rows a warp)
                int a[4];
                gen_rows<KW, 4>(w + i * K, g.lane, x, a);
                if (BYTES) {
                    const uint32_t v = gen_gelu4(s, g.lane, a, bl, i, shift);
                    if (half == 0) st_async_b32(ptx::mapa_u32(at, dest), bar, v);
                } else if (((row0 + i) & 3) == 0) {
                    if (half == 0) st_async_v4(ptx::mapa_u32(at, dest), bar, a[0], a[1], a[2], a[3]);
                } else {
                    st_async_b32(ptx::mapa_u32(at + 4 * half, dest), bar, half ? a[1] : a[0]);
                    st_async_b32(ptx::mapa_u32(at + 4 * (2 + half), dest), bar, half ? a[3] : a[2]);
                }
                i += 4;
            } else if (MOST >= 2 && !BYTES && per - i >= 2) {
                int a[2];
                gen_rows<KW, 2>(w + i * K, g.lane, x, a);
                if (((row0 + i) & 1) == 0) {
                    if (half == 0) st_async_v2(ptx::mapa_u32(at, dest), bar, (uint32_t)a[0], (uint32_t)a[1]);
                } else {
                    st_async_b32(ptx::mapa_u32(at + 4 * half, dest), bar, (uint32_t)(half ? a[1] : a[0]));
                }
                i += 2;
            } else if (!BYTES) {
                int a[1];
                gen_rows<KW, 1>(w + i * K, g.lane, x, a);
                if (half == 0) st_async_b32(ptx::mapa_u32(at, dest), bar, a[0]);
                i++;
            }
        }
        __syncwarp();
        if (g.lane == 0) ptx::mbar_arrive(&s.empty[st]);
        g.ring_it++;
        r += rc;
    }
}

// q, k and v of a layer side by side: three ring stages are held at once, a warp forms NJ sums of each product, and the three waits,
// products and sums overlap.  Up to twelve sums: H 256 5.54 -> 4.97 ms, 384 5.58 -> 5.23 (2 layers, 250 sampled bytes; 128 alike).
// Fifteen (H 640, the widest whose rows fit one chunk) take longer than three products, 7.30 against 7.14 ms: a row of an odd width is
// read by words, and a register spills.
template <int NJ>
constexpr bool GEN_QKV_TOGETHER = NJ <= 4;
template <int NJ>
__device__ __forceinline__ void gen_qkv(GenSmem &s, GenState &g, const int8_t *vec, uint32_t out_off, uint32_t bar_off, int *err) {
    static_assert(8 * NJ * (128 * NJ) <= GEN_CHUNK && GEN_STAGES >= 3, "a block's rows are one chunk each, all held before one is released");
    constexpr int H = NJ * 128, WORDS = NJ % 4 == 0 ? 4 : (NJ % 2 == 0 ? 2 : 1), MSGS = 3 * NJ / WORDS;       // words a message, by its alignment
    int32_t x[NJ];
    gen_load_vec<NJ>(vec, g.lane, x);
    int a[3 * NJ];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t it = g.ring_it + (uint32_t)k;
        gen_wait_ring(s, &s.full[it % GEN_STAGES], (it / GEN_STAGES) & 1, err);
        __syncwarp();
        const int8_t *w = s.ring[it % GEN_STAGES] + g.warp * NJ * H;
#pragma unroll
        for (int i = 0; i < NJ; i++) a[k * NJ + i] = gen_dot<NJ>(w + i * H, g.lane, x);
    }
#pragma unroll
    for (int i = 0; i < 3 * NJ; i++) a[i] = __reduce_add_sync(0xFFFFFFFFu, a[i]);
    const int dest = g.lane & 15, half = g.lane >> 4;
    const uint32_t bar = ptx::mapa_u32(g.smem_base + bar_off, dest), at = ptx::mapa_u32(g.smem_base + out_off + 4 * NJ * (8 * g.rank + g.warp), dest);
    // lanes 0-15 send the even messages, 16-31 the odd ones
#pragma unroll
    for (int m = 0; m < MSGS; m += 2) {
        const int e = m * WORDS, o = (m + 1 < MSGS ? m + 1 : m) * WORDS;
        const uint32_t to = at + 4 * (half ? o / NJ * H + o % NJ : e / NJ * H + e % NJ);
        int v[4];
#pragma unroll
        for (int j = 0; j < WORDS; j++) v[j] = half ? a[o + j] : a[e + j];
        if (o == e && half) continue;
        if (WORDS == 4) st_async_v4(to, bar, v[0], v[1], v[2], v[3]);
        else if (WORDS == 2) st_async_v2(to, bar, v[0], v[1]);
        else st_async_b32(to, bar, v[0]);
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 3; k++)
        if (g.lane == 0) ptx::mbar_arrive(&s.empty[(g.ring_it + (uint32_t)k) % GEN_STAGES]);
    g.ring_it += 3;
}

// Waits for the exchange in flight; its barrier is armed at once for the exchange after the next one (`bytes_after`).
__device__ __forceinline__ void gen_receive(GenSmem &s, GenState &g, uint32_t bytes_after, int *err) {
    uint64_t *bar = &s.ex[g.ex_it & 1];
    gen_wait(s, bar, (g.ex_it >> 1) & 1, err);
    __syncwarp();
    if (g.tid == 0) ptx::mbar_arrive_expect_tx(bar, bytes_after);
    g.ex_it++;
}

// the eight warps' values of a slot
__device__ __forceinline__ void gen_red(const int32_t *r, int (&v)[GEN_WARPS]) {
    static_assert(GEN_WARPS == 8, "two 16-byte reads");
    const int4 a = *reinterpret_cast<const int4 *>(r), b = *reinterpret_cast<const int4 *>(r + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ int gen_red_max(const int32_t *r) {
    int v[GEN_WARPS];
    gen_red(r, v);
    return max(max(max(v[0], v[1]), max(v[2], v[3])), max(max(v[4], v[5]), max(v[6], v[7])));
}
__device__ __forceinline__ int gen_red_sum(const int32_t *r) {
    int v[GEN_WARPS];
    gen_red(r, v);
    return v[0] + v[1] + v[2] + v[3] + v[4] + v[5] + v[6] + v[7];
}
__device__ __forceinline__ int gen_block_max(GenSmem &s, const GenState &g, int slot, int v) {
    v = __reduce_max_sync(0xFFFFFFFFu, v);
    if (g.lane == 0) s.red[slot][g.warp] = v;
    gen_bar();
    return gen_red_max(s.red[slot]);
}

// Four consecutive elements of the row per thread (threads beyond H / 4 carry zeros).
// apply_standard_norm without noise (mgpu.cu:646-678, ns = 0): h = clip((x * w) / mean|x| + b); ends with h in place.
__device__ __forceinline__ void gen_norm(GenSmem &s, const GenState &g, int x4, int w4, int b4, int H) {
    int sum = __reduce_add_sync(0xFFFFFFFFu, abs_sum4((uint32_t)x4, 0));
    const bool in = g.tid < H / 4;
    if (g.lane == 0) s.red[0][g.warp] = sum;
    gen_bar();
    sum = gen_red_sum(s.red[0]);
    int mn = sum / H;
    if (!mn) mn = 1;
    const float rinv = c_rinv_up.v[mn];
    if (in) {
        int o[4];
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = div_small((int)(int8_t)(x4 >> (8 * k)) * (int)(int8_t)(w4 >> (8 * k)), rinv) + (int)(int8_t)(b4 >> (8 * k));
        *reinterpret_cast<uint32_t *>(s.h + 4 * g.tid) = pack_clip8(o[0], o[1], o[2], o[3]);
    }
    gen_bar();
}

// x = adaptive_layer_normalize(x + (product >> shift) + bias) (egg_adaptive_normalize.h:10-103)
__device__ __forceinline__ int gen_finish(GenSmem &s, const GenState &g, int x4, const int32_t *prod, int shift, int b4, int H) {
    int v[4] = {0, 0, 0, 0};
    if (g.tid < H / 4) {
        const int4 a = *reinterpret_cast<const int4 *>(prod + 4 * g.tid);
        v[0] = (a.x >> shift) + (int)(int8_t)x4 + (int)(int8_t)b4;
        v[1] = (a.y >> shift) + (int)(int8_t)(x4 >> 8) + (int)(int8_t)(b4 >> 8);
        v[2] = (a.z >> shift) + (int)(int8_t)(x4 >> 16) + (int)(int8_t)(b4 >> 16);
        v[3] = (a.w >> shift) + (x4 >> 24) + (b4 >> 24);
    }
    const float scale = aln_scale(gen_block_max(s, g, 1, max(max(abs(v[0]), abs(v[1])), max(abs(v[2]), abs(v[3])))));
    return (int)pack_clip8(aln_quant_f(v[0], scale), aln_quant_f(v[1], scale), aln_quant_f(v[2], scale), aln_quant_f(v[3], scale));
}

// trunc(num / den) as C does for a weighted mean num / den of int8 values: the nearest integer to a float estimate (off by less than
// 1e-4) and one exact remainder, where a 64-bit division takes some 500 cycles of every layer.
__device__ __forceinline__ int gen_quotient(long long num, int den) {
    int k = __float2int_rn((float)num / (float)den);
    const long long r = num - (long long)k * den;
    if (k > 0 && r < 0) k--;
    else if (k < 0 && r > 0) k++;
    return k;
}

template <int NJ>
__global__ void __launch_bounds__(GEN_THREADS, 1) generate_kernel(const GenParams p) {
    constexpr int H = NJ * 128, NH = H / 64, V = 256;
    extern __shared__ uint8_t gen_raw[];
    GenSmem &s = *reinterpret_cast<GenSmem *>((reinterpret_cast<uintptr_t>(gen_raw) + 127) & ~uintptr_t(127));
    const int total = p.seed_len + p.gen_len;
    const int8_t *M = p.model;
    const ModelLayout &L = p.L;
    GenState g;
    g.rank = (int)blockIdx.x; g.warp = threadIdx.x >> 5; g.lane = threadIdx.x & 31; g.tid = threadIdx.x;
    g.ring_it = 0; g.ex_it = 0; g.smem_base = ptx::smem_u32(&s);

    for (int i = g.tid; i < 256; i += GEN_THREADS) {
        s.act_lut[i] = p.act_lut[i]; s.exp_lut[i] = p.exp_lut[i]; s.count[i] = 0;
        s.tok[i] = i < p.seed_len ? p.tokens[i] : 0;
    }
    if (g.tid == 0) {
        for (int i = 0; i < GEN_STAGES; i++) { ptx::mbar_init(&s.full[i], 1); ptx::mbar_init(&s.empty[i], GEN_WARPS); }
        ptx::mbar_init(&s.ex[0], 1); ptx::mbar_init(&s.ex[1], 1);
        s.dead = 0;
        ptx::fence_barrier_init();
        ptx::mbar_arrive_expect_tx(&s.ex[0], 4 * H);            // first exchange: MLP activations (bytes), then the down product
        ptx::mbar_arrive_expect_tx(&s.ex[1], 4 * H);
    }
    __syncthreads();
    ptx::cluster_sync_all();
    if (g.tid < p.start) atomicAdd(&s.count[s.tok[g.tid]], 1);          // (a cluster barrier orders the clearing before; start < 256 < block size)
    __syncthreads();

    const int RH = H / GEN_BLOCKS, RU = 4 * H / GEN_BLOCKS, RV = V / GEN_BLOCKS;        // rows per block
    if (g.warp == GEN_WARPS) {
        // ===================== weight stream =====================
        if (g.lane == 0) {
            uint32_t it = 0;
            for (int t = p.start; t < total - 1; t++) {
                gen_stream(s, it, p.w_init_up, g.rank, RU, H, 32, p.err);
                gen_stream(s, it, p.w_init_dn, g.rank, RH, 4 * H, 8, p.err);
                for (int l = 0; l < p.n_layers; l++) {
                    const int8_t *w = p.w_layer0 + l * p.w_layer_stride;
                    for (int k = 0; k < 3; k++) gen_stream(s, it, w + p.w_qkv + (int64_t)k * H * H, g.rank, RH, H, 8, p.err);
                    gen_stream(s, it, w + p.w_o, g.rank, RH, H, 8, p.err);
                    gen_stream(s, it, w + p.w_up, g.rank, RU, H, 32, p.err);
                    gen_stream(s, it, w + p.w_dn, g.rank, RH, 4 * H, 8, p.err);
                }
                if (t >= p.seed_len - 1) gen_stream(s, it, p.w_emb, g.rank, RV, H, 8, p.err);
            }
            if (s.dead) {                          // let copies already in flight land before the block retires
                const uint64_t t0 = ptx::globaltimer();
                while (ptx::globaltimer() - t0 < 200000ull) __nanosleep(1000);
            }
        }
        __syncwarp();
    } else {
        const uint32_t off_qkv = (uint32_t)offsetof(GenSmem, qkv), off_po = (uint32_t)offsetof(GenSmem, po), off_pd = (uint32_t)offsetof(GenSmem, pd);
        const uint32_t off_u = (uint32_t)offsetof(GenSmem, u), off_ao = (uint32_t)offsetof(GenSmem, ao), off_lg = (uint32_t)offsetof(GenSmem, logits);
        auto bar_off = [&]() { return (uint32_t)offsetof(GenSmem, ex) + 8 * (g.ex_it & 1); };
        // this thread's four bytes of a parameter row: loaded a product ahead of their use
        auto row_word = [&](const int8_t *v) { return g.tid < H / 4 ? *reinterpret_cast<const int32_t *>(v + 4 * g.tid) : 0; };
        for (int t = p.start; t < total - 1; t++) {             // after a wait gave up the others fall through: every barrier is still met
            const bool draw = t >= p.seed_len - 1;
            const int tok = s.tok[t];
            if (g.tid == 0) s.count[tok]++;
            int x4 = 0;
            if (g.tid < H / 4) {
                const int e = *reinterpret_cast<const int32_t *>(p.w_emb + (int64_t)tok * H + 4 * g.tid), b = *reinterpret_cast<const int32_t *>(M + L.emb_bias + 4 * g.tid);
                x4 = (int)pack_clip8((int)(int8_t)e + (int)(int8_t)b, (int)(int8_t)(e >> 8) + (int)(int8_t)(b >> 8), (int)(int8_t)(e >> 16) + (int)(int8_t)(b >> 16),
                                     (e >> 24) + (b >> 24));
            }
            // MLP block on the normalised row in s.h (mgpu.cu:708-759); after_u, after_d: bytes of the two exchanges that follow it
            auto mlp = [&](const int8_t *b_up, const int8_t *b_dn, uint32_t after_u, uint32_t after_d) {
                gen_product<NJ, true>(s, g, s.h, RU, 32, off_u, bar_off(), p.err, b_up, p.shift_mlp_up);
                const int bd = row_word(b_dn);
                gen_receive(s, g, after_u, p.err);
                gen_product<4 * NJ, false>(s, g, s.u, RH, 8, off_pd, bar_off(), p.err);
                gen_receive(s, g, after_d, p.err);
                x4 = gen_finish(s, g, x4, s.pd, p.shift_mlp_down, bd, H);
            };
            int nw = row_word(M + L.ln_init), nb = row_word(M + L.ln_init_bias);       // gains and biases of the next norm
            // layer -1 is the embedding's MLP: one copy of the products' code, which a token walks through many times.  At H 128, where the
            // code is short, two copies without the branch in the loop are the faster (224 sampled bytes, 7 layers: 9.92 against 10.03 ms)
            int l = -1;
            if constexpr (NJ == 1) {
                gen_norm(s, g, x4, nw, nb, H);
                nw = row_word(M + L.ln_1); nb = row_word(M + L.ln_1_bias);
                mlp(M + L.mlp_emb_bias_up, M + L.mlp_emb_bias_down, 12 * H, H);
                l = 0;
            }
            for (; l < p.n_layers; l++) {
                const int64_t lH = (int64_t)l * H;
                const bool last = l + 1 == p.n_layers;
                if (NJ == 1 || l >= 0) {
                int8_t *kc = p.kv + ((int64_t)(l * NH + (g.rank < NH ? g.rank : 0)) * 2) * 256 * 64, *vc = kc + 256 * 64;
                const bool head = g.rank < NH;
                gen_norm(s, g, x4, nw, nb, H);
                nw = row_word(M + L.ln_2 + lH); nb = row_word(M + L.ln_2_bias + lH);
                const int4 cs = g.tid < H / 4 ? *reinterpret_cast<const int4 *>(p.rope_lut + t * 64 + (4 * g.tid) % 64) : make_int4(0, 0, 0, 0);
                if constexpr (GEN_QKV_TOGETHER<NJ>) gen_qkv<NJ>(s, g, s.h, off_qkv, bar_off(), p.err);
                else
                    for (int k = 0; k < 3; k++) gen_product<NJ, false>(s, g, s.h, RH, 8, off_qkv + 4 * k * H, bar_off(), p.err);
                // this thread's context row of K and its pieces of V: on their way during the exchange.  (Ahead of the norm
                // its shared-memory accesses waited behind them, 900 cycles a layer)
                const int d4 = g.lane & 15, c0 = 2 * g.warp + (g.lane >> 4);
                int4 kr[4];
                int32_t vr[16];
                if (head) {
                    if (g.tid < t) {
#pragma unroll
                        for (int j = 0; j < 4; j++) kr[j] = *reinterpret_cast<const int4 *>(kc + g.tid * 64 + 16 * j);
                    }
#pragma unroll
                    for (int i = 0; i < 16; i++) vr[i] = c0 + 16 * i < t ? *reinterpret_cast<const int32_t *>(vc + (c0 + 16 * i) * 64 + 4 * d4) : 0;
                }
                gen_receive(s, g, 4 * H, p.err);               // after the attention exchange: the output product
                // integer RoPE on q and k (apply_rope_integer, mgpu.cu:624-644), maxima of q, k, v
                int qv[3][4];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    int4 a = make_int4(0, 0, 0, 0);
                    if (g.tid < H / 4) {
                        a = *reinterpret_cast<const int4 *>(s.qkv + k * H + 4 * g.tid);
                        if (k < 2) {
                            const long long half_ulp = 1ll << (p.rope_bit - 1);
                            const int e0 = a.x, o0 = a.y, e1 = a.z, o1 = a.w;
                            a.x = ptx::shr64_lo(ptx::mad_wide(-o0, cs.y, ptx::mad_wide(e0, cs.x, half_ulp)), p.rope_bit);
                            a.y = ptx::shr64_lo(ptx::mad_wide(o0, cs.x, ptx::mad_wide(e0, cs.y, half_ulp)), p.rope_bit);
                            a.z = ptx::shr64_lo(ptx::mad_wide(-o1, cs.w, ptx::mad_wide(e1, cs.z, half_ulp)), p.rope_bit);
                            a.w = ptx::shr64_lo(ptx::mad_wide(o1, cs.z, ptx::mad_wide(e1, cs.w, half_ulp)), p.rope_bit);
                        }
                    }
                    qv[k][0] = a.x; qv[k][1] = a.y; qv[k][2] = a.z; qv[k][3] = a.w;
                    const int m = __reduce_max_sync(0xFFFFFFFFu, max(max(abs(a.x), abs(a.y)), max(abs(a.z), abs(a.w))));
                    if (g.lane == 0) s.red[2 + k][g.warp] = m;
                }
                gen_bar();
                if (head) {
                    if (g.tid / 16 == g.rank && g.tid < H / 4) {
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            const float sc = aln_scale(gen_red_max(s.red[2 + k]));
                            const uint32_t w = pack_clip8(aln_quant_f(qv[k][0], sc), aln_quant_f(qv[k][1], sc), aln_quant_f(qv[k][2], sc), aln_quant_f(qv[k][3], sc));
                            const int o = 4 * (g.tid & 15);
                            *reinterpret_cast<uint32_t *>((k == 0 ? s.q8 : (k == 1 ? s.k8 : s.v8)) + o) = w;
                            if (k) *reinterpret_cast<uint32_t *>((k == 1 ? kc : vc) + t * 64 + o) = w;
                        }
                    }
                    gen_bar();
                    // scores and weights (mgpu.cu:795-815), one context per thread
                    int sc = INT_MIN;
                    if (g.tid <= t) {
                        if (g.tid == t) {
#pragma unroll
                            for (int j = 0; j < 4; j++) kr[j] = *reinterpret_cast<const int4 *>(s.k8 + 16 * j);
                        }
                        sc = 0;
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const int4 q = *reinterpret_cast<const int4 *>(s.q8 + 16 * j);
                            sc = __dp4a(q.x, kr[j].x, sc); sc = __dp4a(q.y, kr[j].y, sc); sc = __dp4a(q.z, kr[j].z, sc); sc = __dp4a(q.w, kr[j].w, sc);
                        }
                    }
                    const int mx = gen_block_max(s, g, 5, sc);
                    int w = 0;
                    if (g.tid <= t) {
                        int idx = (mx >> p.shift_attn) - (sc >> p.shift_attn);
                        w = s.exp_lut[idx < 0 ? 0 : (idx > 255 ? 255 : idx)];
                    }
                    s.wt[g.tid] = w;
                    // at most 256 weights of 2^20 each
                    const int wsum = __reduce_add_sync(0xFFFFFFFFu, w);
                    if (g.lane == 0) s.red[6][g.warp] = wsum;
                    gen_bar();
                    // Σ w·v (mgpu.cu:816-824): 16 contexts per thread stay below 16 * 2^20 * 127 < 2^31, wider sums in 64 bits
                    if (((t - c0) & 15) == 0 && t >= c0) {
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            if (c0 + 16 * i == t) vr[i] = *reinterpret_cast<const int32_t *>(s.v8 + 4 * d4);
                    }
                    int a[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const int wi = s.wt[c0 + 16 * i];
                        a[0] += wi * (int)(int8_t)vr[i]; a[1] += wi * (int)(int8_t)(vr[i] >> 8); a[2] += wi * (int)(int8_t)(vr[i] >> 16); a[3] += wi * (vr[i] >> 24);
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const long long b = (long long)a[k] + (long long)__shfl_xor_sync(0xFFFFFFFFu, a[k], 16);
                        if (g.lane < 16) s.part[g.warp][4 * d4 + k] = b;
                    }
                    gen_bar();
                    if (g.warp < 2) {
                        const int d = 32 * g.warp + g.lane;
                        long long wv = 0;
#pragma unroll
                        for (int i = 0; i < GEN_WARPS; i++) wv += s.part[i][d];
                        const int tot = gen_red_sum(s.red[6]);
                        const uint32_t o = (uint32_t)gen_quotient(wv, tot ? tot : 1) & 0xFF;
                        // lane 4i + j -> byte j of word i; eight words go to sixteen blocks
                        uint32_t word = o << (8 * (g.lane & 3));
                        word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
                        word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
                        const int hf = g.lane >> 4, dest = g.lane & 15;
                        const uint32_t x0 = __shfl_sync(0xFFFFFFFFu, word, 16 * hf), x1 = __shfl_sync(0xFFFFFFFFu, word, 16 * hf + 4);
                        const uint32_t x2 = __shfl_sync(0xFFFFFFFFu, word, 16 * hf + 8), x3 = __shfl_sync(0xFFFFFFFFu, word, 16 * hf + 12);
                        st_async_v4(ptx::mapa_u32(g.smem_base + off_ao + g.rank * 64 + 32 * g.warp + 16 * hf, dest), ptx::mapa_u32(g.smem_base + bar_off(), dest),
                                    (int)x0, (int)x1, (int)x2, (int)x3);
                    }
                }
                gen_receive(s, g, 4 * H, p.err);               // after the output product: the MLP activations
                gen_product<NJ, false>(s, g, s.ao, RH, 8, off_po, bar_off(), p.err);
                gen_receive(s, g, 4 * H, p.err);               // after the activations: the down product
                x4 = gen_finish(s, g, x4, s.po, p.shift_out, 0, H);
                }
                gen_norm(s, g, x4, nw, nb, H);
                nw = row_word(last ? M + L.ln_f : M + L.ln_1 + lH + H); nb = row_word(last ? M + L.ln_f_bias : M + L.ln_1_bias + lH + H);
                // what follows this block: the next layer's q|k|v and attention; at the end the logits (when drawing) and the next
                // token's first two exchanges
                const uint32_t e1 = !last ? 12 * H : (draw ? 4 * V : 4 * H), e2 = !last ? H : 4 * H;
                mlp(M + (l < 0 ? L.mlp_emb_bias_up : L.mlp_bias_up + 4 * lH), M + (l < 0 ? L.mlp_emb_bias_down : L.mlp_bias_down + lH), e1, e2);
            }

            if (draw) {
                // head on the tied embedding, presence penalty, temperature, min-p filter, weighted draw
                gen_norm(s, g, x4, nw, nb, H);
                gen_product<NJ, false>(s, g, s.h, RV, 8, off_lg, bar_off(), p.err);
                gen_receive(s, g, 4 * H, p.err);
                const int lg = (s.logits[g.tid] >> p.shift_logit) - s.count[g.tid] * p.penalty_int;
                const int mx = gen_block_max(s, g, 7, lg);
                const int scaled = (int)__fdiv_rn((float)(lg - mx), p.temp);      // (int32_t)(shifted / temp)
                int e = 0;
                if (!p.filter || scaled >= p.min_p_limit) { int idx = -scaled; idx = idx < 0 ? 0 : (idx > 255 ? 255 : idx); e = s.exp_lut[idx]; }
                s.wt[g.tid] = e;
                if (g.tid == 0) s.sel = 0;
                gen_bar();
                // the reference's block scan runs thread-major: thread i owns v = i, i + B, ... (B = its block size)
                const int B = p.scan_block < V ? p.scan_block : V, per = V / B;
                const int v = g.tid / per + B * (g.tid % per);
                const int mine = s.wt[v];
                int run = mine;                                // inclusive prefix over the warp's 32 positions
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int up = __shfl_up_sync(0xFFFFFFFFu, run, o);
                    if (g.lane >= o) run += up;
                }
                if (g.lane == 31) s.red[0][g.warp] = run;
                gen_bar();
                int sum = 0;
#pragma unroll
                for (int i = 0; i < GEN_WARPS; i++) {
                    const int w = s.red[0][i];
                    if (i < g.warp) run += w;
                    sum += w;
                }
                const uint32_t r = hash_rng(p.seed + (uint32_t)t * 555u, 0);
                const int thresh = sum > 0 ? (int)(r % (uint32_t)sum) : 0;
                if (run > thresh && run - mine <= thresh) s.sel = v;
                gen_bar();
                if (g.tid == 0) {
                    s.tok[t + 1] = (uint8_t)s.sel;
                    if (g.rank == 0) p.tokens[t + 1] = (uint8_t)s.sel;
                }
            }
            gen_bar();
        }
    }
    __syncwarp();
    __syncthreads();
    ptx::cluster_sync_all();                                   // no block retires while a peer may still write into it
}

// The cache's layout from rows of k and v as the evaluation's projections leave them; one block per token, a few KB each.
__global__ void kv_gather_kernel(const int8_t *k, const int8_t *v, int H, int8_t *kv) {
    chain_next();
    chain_wait();
    const int t = blockIdx.x;
    for (int d = threadIdx.x * 16; d < H; d += blockDim.x * 16) {
        int8_t *o = kv + ((int64_t)(d >> 6) * 2 * 256 + t) * 64 + (d & 63);
        *reinterpret_cast<int4 *>(o) = *reinterpret_cast<const int4 *>(k + (int64_t)t * H + d);
        *reinterpret_cast<int4 *>(o + 256 * 64) = *reinterpret_cast<const int4 *>(v + (int64_t)t * H + d);
    }
}
int launch_kv_gather(cudaStream_t st, const int8_t *k, const int8_t *v, int H, int count, int8_t *kv) {
    EGG_CUDA(launch_chained(kv_gather_kernel, count, 64, 0, st, k, v, H, kv));
    return EGG_OK;
}

template <int NJ>
static int launch_generate_one(cudaStream_t st, const GenParams &p) {
    static bool attr_set[EGG_MAX_DEVICES] = {};
    const int dev = current_device_slot();
    auto kern = generate_kernel<NJ>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(GEN_BLOCKS);
    cfg.blockDim = dim3(GEN_THREADS);
    cfg.dynamicSmemBytes = sizeof(GenSmem) + 128;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = GEN_BLOCKS; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    if (!attr_set[dev]) {
        EGG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes));
        EGG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        int n = 0;
        EGG_CUDA(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
        if (n < 1) { set_error("a cluster of %d blocks does not fit this device", GEN_BLOCKS); return EGG_E_CUDA; }
        attr_set[dev] = true;
    }
    EGG_CUDA(cudaLaunchKernelEx(&cfg, kern, p));
    return EGG_OK;
}

int launch_generate(cudaStream_t st, const GenParams &p) {
    switch (p.H) {
        case 128: return launch_generate_one<1>(st, p);
        case 256: return launch_generate_one<2>(st, p);
        case 384: return launch_generate_one<3>(st, p);
        case 512: return launch_generate_one<4>(st, p);
        case 640: return launch_generate_one<5>(st, p);
        case 768: return launch_generate_one<6>(st, p);
        case 896: return launch_generate_one<7>(st, p);
        case 1024: return launch_generate_one<8>(st, p);
    }
    set_error("hidden_dim %d cannot be sampled", p.H);
    return EGG_E_INVALID;
}

}  // namespace egg
