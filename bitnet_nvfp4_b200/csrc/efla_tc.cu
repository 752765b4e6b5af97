// EFLA scan over whole sequences of 33 to 128 tokens, heads of 64, half inputs and output, method 1, zero initial state: the closed form on the
// fifth-generation tensor cores.
//
// With K, Q, V the rows of one (sequence, head), G = K K^T and a_t the token's step size, the recurrence is
//     (I + diag(a) strict(G)) U = diag(a) V,      Y = diag(q_inv) (Q K^T, s <= t) U
// (reference recurrence: src/efla_lm_kernels.cu:590-726). The two 128 x 128 x 64 products are one tcgen05 tile each; what is left for mma.sync
// is the blocked forward substitution and Y = P U, 36 blocks of 16 x 16 each. The kernel that carries the 64 x 64 state from chunk to chunk
// of 16 tokens is bound by the latency of a chunk's chain (4700 cycles, eight of them); here the chain between blocks is two products. 4 to 32 sequences of
// 8 heads x 128 tokens 13.4 -> 6.4 and 13.8 -> 8.8 us, 8192 sequences 1.05 to 1.2 -> 0.93 ms (69 % of the shared-memory wavefronts: four warps each read all
// blocks; tensor pipe 44 %), 4096 x 64 tokens 280 -> 196 us. Nothing is rounded to fp16 between chunks: the operands of the block products (a G, T - I, a V, U, P)
// are halves and all sums are fp32, so the result is nearer to the recurrence in float64 (relative error at 128 tokens 4.3e-4 instead of 5.0e-4).
//
// Keys far from unit length would leave the halves' range: a G and P grow with the ratio of two keys' lengths, U falls with its key's square. Where |k_s|
// is below 2^-6 or from 2^6 on, the unknown is s U_s with s a power of two next to |k_s|: rows of a G and a V take the factor s_t, columns of a G and of P 1 / s_s, all in
// fp32 and exact, so that no coefficient exceeds 64 and s U is as large as y. Tokens in between have s = 1, and blocks of them skip the products. (128 tokens, relative error with s = 1
// throughout: |k| near 8e-5 1.8e-3, near 800 1.2e-2, and infinities from |k| = 65504 on. What it costs keys of ordinary length: 32 sequences of 8 heads 7.4 -> 7.75 us,
// 8192 sequences 911 -> 919, 4096 x 64 tokens the same; where all blocks are scaled 1170.)
//
// Sequences of at most 64 tokens share a tile: R = 8 / NB of them (NB blocks of 16 tokens each), whose products across sequences are not read.
//
// One CTA (288 threads, two per SM) walks units of R sequences of one head, three roles one behind the other:
//   warp 8     TMA tiles of Q, K, V (up to 128 tokens x 64 halves, 128B swizzle) and the two tcgen05 products into tensor memory
//   warps 0-3  a thread per token: the queries' norms (mma.sync on the diagonal 16 x 16 blocks, while the products run), the keys' norms (G's diagonal) and
//              step sizes, T - I with T the inverses of the diagonal blocks of I + a G (forward substitution in fp32), and -a G and q_inv Q K^T, all as
//              halves in shared memory, 32 tokens' rows at a time: a unit's first rows follow while the last ones of the unit before are still read
//   warps 4-7  16 value columns each: X_i = a_i V_i + sum_{j<i} (-a G)_ij U_j, U_i = X_i + (T - I) X_i, Y_i = sum_{j<=i} P_ij U_j on transposed operands, so
//              that U's accumulator fragments are the next products' A fragments; Y takes V's place in shared memory and leaves by TMA.

#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "kernels.h"
#include "mma_sync.cuh"
#include "tcgen05.cuh"

namespace bnf4 {

namespace {

constexpr int kTok = 128;                     // tokens of a tile
constexpr int kTileBytes = kTok * 128;        // 64 halves per row
constexpr int kBlocks = kTok / 16;
constexpr int kTriBytes = kBlocks * (kBlocks + 1) / 2 * 512;  // blocks of 16 x 16 halves on and below the diagonal
constexpr int kThreads = 288;

constexpr int kSmemQ = 0;
constexpr int kSmemK = kSmemQ + kTileBytes;
constexpr int kSmemV = kSmemK + kTileBytes;   // two buffers
constexpr int kSmemL = kSmemV + 2 * kTileBytes;   // -a G below the diagonal blocks, (T - I)^T in them
constexpr int kSmemP = kSmemL + kTriBytes;
constexpr int kDBlock = 272;                  // floats of a diagonal block of -a G, by columns (and 16 for the banks)
constexpr int kSmemD = kSmemP + kTriBytes;
constexpr int kSmemAlpha = kSmemD + kBlocks * kDBlock * 4;
constexpr int kSmemKey = kSmemAlpha + kTok * 4;  // 1 / s of the tokens, and whether 32 of them have another s than 1
constexpr int kSmemBar = kSmemKey + kTok * 4 + 16;
constexpr int kBarTriFree = 96;               // of the barriers: see the kernel
constexpr int kSmemAlloc = kSmemBar + 256 + 1024;
static_assert(2 * (kSmemAlloc + 1024) <= 233472, "two CTAs per SM");

constexpr float kKeyLow = 1.0f / 4096.0f, kKeyHigh = 4096.0f;  // squared lengths of keys with s = 1

constexpr int kTmemCols = 256;  // G | Q K^T
constexpr uint32_t kIdescF16 = (1u << 4) | (static_cast<uint32_t>(kTok >> 3) << 17) | (static_cast<uint32_t>(kTok >> 4) << 24);  // f16 x f16 -> fp32, K-major

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Waits for the 128 threads that meet at barrier 1. Does x hold for all of them?
__device__ __forceinline__ bool all_of_barrier1(bool x) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"(static_cast<uint32_t>(x))
        : "memory");
    return all != 0;
}

__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// Blocks of 16 x 16 halves, block (i, j <= i) at tri(i, j): four 8 x 8 matrices of 128 bytes, (row half, column half) at 128 * row half + 256 * column
// half. A row of eight halves is one 16-byte piece, so the token-per-lane stores and every ldmatrix phase touch 128 contiguous bytes.
__device__ __forceinline__ uint32_t tri(int i, int j) { return static_cast<uint32_t>(i * (i + 1) / 2 + j) * 512u; }

// What a token's thread leaves for the substitution, in its warp's 32 rows of L, T and P. FAR: columns take their keys' scales (in the chunks whose bit is set).
struct TokenRows {
    uint32_t smem_base, trow;  // the warp's lanes of tensor memory
    int first_chunk;           // 32 columns at a time, from the one in which the warp's first sequence starts
    uint32_t far, n;           // n: units before this one
    float alpha, qinv;
};
// rg: the chunk of G on the diagonal. Returns false when a wait has expired.
template <bool FAR>
__device__ __forceinline__ bool token_rows(const TokenRows& a, uint32_t (&rg)[32]) {
    const int w = static_cast<int>(threadIdx.x) >> 5, lane = threadIdx.x & 31, t = 32 * w + lane, half = lane >> 4;
    const int bi = 2 * w + half;  // this token's block row
    const uint32_t lrow = static_cast<uint32_t>((lane >> 3) & 1) * 128u + static_cast<uint32_t>(lane & 7) * 16u;  // this token's row in its blocks
    const uint32_t l_row = a.smem_base + kSmemL + tri(bi, 0) + lrow, p_row = a.smem_base + kSmemP + tri(bi, 0) + lrow;
    const uint32_t dcol = a.smem_base + kSmemD + static_cast<uint32_t>(bi * kDBlock * 4);  // the token's diagonal block of -a G by columns
    const float alpha = a.alpha;
    auto scale_columns = [&](uint32_t (&r)[32], int cc) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const float4 f = ld_shared_f4(a.smem_base + kSmemKey + 128 * cc + 4 * j);
            r[j] = __float_as_uint(__uint_as_float(r[j]) * f.x);
            r[j + 1] = __float_as_uint(__uint_as_float(r[j + 1]) * f.y);
            r[j + 2] = __float_as_uint(__uint_as_float(r[j + 2]) * f.z);
            r[j + 3] = __float_as_uint(__uint_as_float(r[j + 3]) * f.w);
        }
    };
    // 32 scaled columns of this token's row as halves: four pieces of eight, from block column 2 cc on
    auto store_row = [&](const float (&x)[32], uint32_t row, int cc, bool left, bool right) {
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8)
            if (c8 < 2 ? left : right)
                st_shared_v4(row + static_cast<uint32_t>(2 * cc + (c8 >> 1)) * 512u + (c8 & 1) * 256u, pack_half2(x[8 * c8], x[8 * c8 + 1]),
                             pack_half2(x[8 * c8 + 2], x[8 * c8 + 3]), pack_half2(x[8 * c8 + 4], x[8 * c8 + 5]), pack_half2(x[8 * c8 + 6], x[8 * c8 + 7]));
    };
    auto scaled = [](float f, const uint32_t (&r)[32], float (&x)[32]) {
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
            const float2 y = __fmul2_rn(make_float2(f, f), make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])));
            x[j] = y.x;
            x[j + 1] = y.y;
        }
    };
    if (FAR && ((a.far >> w) & 1u)) scale_columns(rg, w);
    uint32_t left[8], hv[8];  // the left half of the diagonal chunk and T - I, as halves
#pragma unroll
    for (int j = 0; j < 8; ++j) left[j] = pack_half2(-alpha * __uint_as_float(rg[2 * j]), -alpha * __uint_as_float(rg[2 * j + 1]));
    __syncwarp();  // (the previous unit's reads are done)
#pragma unroll
    for (int s = 0; s < 16; ++s) st_shared(dcol + 64 * s + 4 * (lane & 15), __float_as_uint(-alpha * __uint_as_float(half ? rg[16 + s] : rg[s])));
    __syncwarp();
    {
        // T = (I + a G)^-1 of the token's block by forward substitution: lane c of a half owns column c; a finished element goes
        // into all later ones at once
        const int c = lane & 15;
        float col[16];
#pragma unroll
        for (int s = 0; s < 16; ++s) col[s] = s == c ? 1.0f : 0.0f;
#pragma unroll
        for (int s = 0; s < 15; ++s)
#pragma unroll
            for (int t4 = (s + 1) / 4 * 4; t4 < 16; t4 += 4) {
                const float4 lv = ld_shared_f4(dcol + 64 * s + 4 * t4);
                if (t4 > s) col[t4] = fmaf(lv.x, col[s], col[t4]);
                if (t4 + 1 > s) col[t4 + 1] = fmaf(lv.y, col[s], col[t4 + 1]);
                if (t4 + 2 > s) col[t4 + 2] = fmaf(lv.z, col[s], col[t4 + 2]);
                if (t4 + 3 > s) col[t4 + 3] = fmaf(lv.w, col[s], col[t4 + 3]);
            }
#pragma unroll
        for (int e = 0; e < 8; ++e) hv[e] = pack_half2(2 * e == c ? 0.0f : col[2 * e], 2 * e + 1 == c ? 0.0f : col[2 * e + 1]);
    }
    if (a.n > 0 && !__all_sync(0xffffffffu, mbar_wait(a.smem_base + kSmemBar + kBarTriFree + 8 * w, (a.n - 1) & 1u, 17))) return false;
    st_shared(a.smem_base + kSmemAlpha + 4 * t, __float_as_uint(alpha));
    const uint32_t d = l_row + static_cast<uint32_t>(bi) * 512u;  // row c of (T - I)^T
    st_shared_v4(d, hv[0], hv[1], hv[2], hv[3]);
    st_shared_v4(d + 256u, hv[4], hv[5], hv[6], hv[7]);
    if (half == 1) {
        st_shared_v4(d - 512u, left[0], left[1], left[2], left[3]);
        st_shared_v4(d - 256u, left[4], left[5], left[6], left[7]);
    }
    for (int cc = a.first_chunk; cc < w; ++cc) {
        uint32_t rc[32], rp[32];
        float x[32];
        tmem_ld32(a.trow + 32 * cc, rc);
        tmem_ld32(a.trow + 128 + 32 * cc, rp);
        tmem_ld_wait();
        if (FAR && ((a.far >> cc) & 1u)) {
            scale_columns(rc, cc);
            scale_columns(rp, cc);
        }
        scaled(-alpha, rc, x);
        store_row(x, l_row, cc, true, true);
        scaled(a.qinv, rp, x);
        store_row(x, p_row, cc, true, true);
    }
    uint32_t rp[32];
    float x[32];
    tmem_ld32(a.trow + 128 + 32 * w, rp);
    tmem_ld_wait();
    if (FAR && ((a.far >> w) & 1u)) scale_columns(rp, w);
    scaled(a.qinv, rp, x);
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = j <= lane ? x[j] : 0.0f;
    store_row(x, p_row, w, true, half == 1);
    return true;
}
// (a function of its own: the products and their registers stay out of the usual path)
__device__ __noinline__ bool token_rows_far(const TokenRows a) {
    uint32_t rg[32];
    tmem_ld32(a.trow + 32 * (threadIdx.x >> 5), rg);
    tmem_ld_wait();
    return token_rows<true>(a, rg);
}

template <int NB>
__global__ void __launch_bounds__(kThreads, 2) efla_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                              const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o,
                                                              const EflaParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const uint32_t bar_qk = smem_base + kSmemBar;    // Q and K have arrived
    const uint32_t bar_qk_free = bar_qk + 8;         // products and norms have read them (1 + 4)
    const uint32_t bar_v = bar_qk_free + 8;          // V has arrived (2)
    const uint32_t bar_v_free = bar_v + 16;          // Y has left V's buffer (2)
    const uint32_t bar_prod = bar_v_free + 16;       // products complete
    const uint32_t bar_prod_free = bar_prod + 8;     // tensor memory has been read (4)
    const uint32_t bar_tri = bar_prod_free + 8;      // L, T, P and the step sizes of 32 tokens are there (4 barriers)
    const uint32_t bar_tri_free = bar_qk + kBarTriFree;  // and have been read (4 x 4)
    const uint32_t bar_key = bar_tri_free + 32;      // the keys' scales are there (the warps with tokens)
    const uint32_t tmem_slot = bar_key + 8;
    volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + kSmemBar + (tmem_slot - bar_qk));

    if (threadIdx.x == 0) {
        mbar_init(bar_qk, 1);
        mbar_init(bar_qk_free, 5);
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_v + 8 * b, 1);
            mbar_init(bar_v_free + 8 * b, 1);
        }
        mbar_init(bar_prod, 1);
        mbar_init(bar_prod_free, 4);
        mbar_init(bar_key, (kBlocks / NB * NB + 1) / 2);
        for (int b = 0; b < 4; ++b) {
            mbar_init(bar_tri + 8 * b, 1);
            mbar_init(bar_tri_free + 8 * b, 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_gen;
    pdl_wait();

    constexpr int R = kBlocks / NB, kUsed = NB * R;  // sequences and blocks of a unit
    const unsigned heads = static_cast<unsigned>(p.heads);
    const unsigned total = (static_cast<unsigned>(p.seqs) + R - 1) / R * heads;  // below 2^31 (checked by the host)
    bool ok = true;

    if (warp == 8) {
        // ------------------------------ loads and products ------------------------------
        const uint64_t qdesc = smem_desc(smem_base + kSmemQ, 16, 1024, kLayoutSw128), kdesc = smem_desc(smem_base + kSmemK, 16, 1024, kLayoutSw128);
        constexpr uint32_t bytes = kUsed * 16u * 128u;  // (boxes of 16 NB tokens of R sequences; tokens past T and sequences past the last arrive as zeros)
        auto load_qk = [&](unsigned u) {
            const unsigned su = u / heads;
            const int seq = static_cast<int>(su * R), x = static_cast<int>(u - su * heads) * 64;
            if (elect_one()) {
                mbar_expect_tx(bar_qk, 2 * bytes);
                tma_load_3d(smem_base + kSmemK, &map_k, x, 0, seq, bar_qk);
                tma_load_3d(smem_base + kSmemQ, &map_q, x, 0, seq, bar_qk);
            }
            __syncwarp();
        };
        auto load_v = [&](unsigned u, uint32_t buf) {
            const unsigned su = u / heads;
            const int seq = static_cast<int>(su * R), x = static_cast<int>(u - su * heads) * 64;
            if (elect_one()) {
                mbar_expect_tx(bar_v + 8 * buf, bytes);
                tma_load_3d(smem_base + kSmemV + buf * kTileBytes, &map_v, x, 0, seq, bar_v + 8 * buf);
            }
            __syncwarp();
        };
        if (blockIdx.x < total) {
            load_qk(blockIdx.x);
            load_v(blockIdx.x, 0);
        }
        uint32_t n = 0;
        for (unsigned u = blockIdx.x; u < total && ok; u += gridDim.x, ++n) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar_qk, n & 1u, 11));
            if (ok && n > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar_prod_free, (n - 1) & 1u, 12));
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int j = 0; j < 4; ++j) tc_mma_f16(tmem_base, kdesc + 2 * j, kdesc + 2 * j, kIdescF16, j > 0 ? 1u : 0u);
#pragma unroll
                for (int j = 0; j < 4; ++j) tc_mma_f16(tmem_base + 128, qdesc + 2 * j, kdesc + 2 * j, kIdescF16, j > 0 ? 1u : 0u);
                tc_commit(bar_qk_free);
                tc_commit(bar_prod);
            }
            __syncwarp();
            const unsigned next = u + gridDim.x;
            if (next < total) {
                ok = __all_sync(0xffffffffu, mbar_wait(bar_qk_free, n & 1u, 13));
                if (!ok) break;
                load_qk(next);
                const uint32_t buf = (n + 1) & 1u;
                if (n > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar_v_free + 8 * buf, ((n - 1) >> 1) & 1u, 14));  // (unit n - 1 had this buffer)
                if (!ok) break;
                load_v(next, buf);
            }
        }
        pdl_trigger();
    } else if (warp < 4) {
        // ------------------------------ a thread per token ------------------------------
        const int w = warp, t = 32 * w + lane, half = lane >> 4;
        const bool rows = 2 * w < kUsed;  // this warp has tokens
        const int tok = t % (16 * NB);    // and its place in its sequence
        const unsigned sub = static_cast<unsigned>(t / (16 * NB));
        const int first_chunk = (2 * w - 2 * w % NB) / 2;  // 32 columns at a time, from the one in which the warp's first sequence starts
        const uint32_t key_sh = smem_base + kSmemKey, far_sh = key_sh + kTok * 4;
        // ldmatrix rows of the two 16-token blocks (128B swizzle): matrices (tokens 0-7 | d 0-7), (0-7 | 8-15), (8-15 | 0-7), (8-15 | 8-15)
        const uint32_t lm = static_cast<uint32_t>(32 * w + (lane >> 4) * 8 + (lane & 7)) * 128u + static_cast<uint32_t>(((lane >> 3) & 1) ^ (lane & 7)) * 16u;
        // squared norms of this warp's 32 queries from the diagonals of Q Q^T, handed to the token's thread
        auto query_norm = [&]() {
            float c[2][2][4];  // [block][token half][..]
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    uint32_t f[4];
                    ldmatrix_x4(f, (smem_base + kSmemQ + lm + static_cast<uint32_t>(b) * 2048u) ^ static_cast<uint32_t>(ks * 32));
                    if (ks == 0) {
                        mma_f16_16816_zero(c[b][0], f[0], f[2], f[1], f[3], f[0], f[1]);
                        mma_f16_16816_zero(c[b][1], f[0], f[2], f[1], f[3], f[2], f[3]);
                    } else {
                        mma_f16_16816(c[b][0], f[0], f[2], f[1], f[3], f[0], f[1]);
                        mma_f16_16816(c[b][1], f[0], f[2], f[1], f[3], f[2], f[3]);
                    }
                }
            // tokens g and g + 8 of a block lie in the lane 4 g + g / 2, columns g and g + 8
            const bool odd = (lane >> 2) & 1;
            const int tk = lane & 7, src = 4 * tk + (tk >> 1);
            float mine = 0.0f;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const float lo = __shfl_sync(0xffffffffu, odd ? c[b][0][1] : c[b][0][0], src), hi = __shfl_sync(0xffffffffu, odd ? c[b][1][3] : c[b][1][2], src);
                if (half == b) mine = (lane & 8) ? hi : lo;
            }
            return mine;
        };
        uint32_t n = 0;
        float braw = 0.0f;
        auto fetch_beta = [&](unsigned u) {
            const unsigned seq = u / heads * R + sub;
            if (u < total && tok < p.T && seq < static_cast<unsigned>(p.seqs)) braw = p.beta_raw[(static_cast<size_t>(seq) * p.T + tok) * p.ld_beta];
        };
        fetch_beta(blockIdx.x);
        for (unsigned u = blockIdx.x; u < total && ok; u += gridDim.x, ++n) {
            const float logit = braw + efla_seq_bias(p, min(u / heads * R + sub, static_cast<unsigned>(p.seqs) - 1u));
            fetch_beta(u + gridDim.x);
            ok = __all_sync(0xffffffffu, mbar_wait(bar_qk, n & 1u, 15));
            if (!ok) break;
            float qinv = 0.0f;
            if (rows) qinv = rsqrtf(query_norm() + p.eps);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_qk_free);
            ok = __all_sync(0xffffffffu, mbar_wait(bar_prod, n & 1u, 16));
            if (!ok) break;
            tc_fence_after();
            const uint32_t trow = tmem_base + (static_cast<uint32_t>(32 * w) << 16);
            if (rows) {
                // the chunk of G on the diagonal: block (2 w + 1, 2 w) in its lower left and two diagonal blocks; G_tt is the key's squared norm
                uint32_t rg[32];
                tmem_ld32(trow + 32 * w, rg);
                tmem_ld_wait();
                uint32_t pick[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t lo = half ? rg[16 + j] : rg[j], hi = half ? rg[24 + j] : rg[8 + j];
                    pick[j] = (lane & 8) ? hi : lo;
                }
#pragma unroll
                for (int k = 4; k > 0; k >>= 1)
#pragma unroll
                    for (int j = 0; j < k; ++j) pick[j] = (lane & k) ? pick[j + k] : pick[j];
                const float kss = __uint_as_float(pick[0]);
                // the key's scale: the next unit's are written behind its products, which wait for every warp to have read this one's
                const bool off = t < 16 * kUsed && !(kss >= kKeyLow && kss < kKeyHigh) && kss > 0.0f && kss <= FLT_MAX;  // (what lies behind the last block is no token)
                uint32_t far = __any_sync(0xffffffffu, off) ? 1u << w : 0u;  // bit c: tokens 32 c .. have another s than 1
                float key = 1.0f;
                if (far) {
                    float key_inv = 1.0f;
                    if (off) {
                        const int e = (static_cast<int>(__float_as_uint(kss) >> 23) - 127) >> 1;
                        key = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
                        key_inv = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
                    }
                    st_shared(key_sh + 4 * t, __float_as_uint(key_inv));
                }
                if (lane == 0) st_shared(far_sh + 4 * w, far);
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_key);
                const float lambda = kss < p.eps ? p.eps : kss;
                // sigmoid and the final quotient with the fast exponential / division (about 2 ulp each: far below the fp16
                // rounding of every operand alpha touches); expm1f keeps its accuracy for small beta * lambda
                const float beta = __fdividef(1.0f, 1.0f + __expf(-logit));
                const float alpha = tok < p.T ? __fdividef(-expm1f(-(beta * lambda)), lambda + p.eps) * key : 0.0f;  // a s
                if (w > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_key, n & 1u, 20));
                    if (!ok) break;
                    const float4 f = ld_shared_f4(far_sh);
                    far |= (__float_as_uint(f.x) | __float_as_uint(f.y) | __float_as_uint(f.z)) & ((1u << w) - 1u);
                }
                const TokenRows r = {smem_base, trow, first_chunk, far, n, alpha, qinv};
                ok = __builtin_expect(far, 0) ? token_rows_far(r) : token_rows<false>(r, rg);
                if (!ok) break;
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bar_prod_free);
                mbar_arrive(bar_tri + 8 * w);
            }
        }
    } else {
        // ------------------------------ substitution and output: 16 value columns per warp ------------------------------
        const int c = warp - 4, tq = lane & 3, j4 = lane >> 3, r8 = lane & 7;
        // V read and Y written through transposing matrix loads / stores: matrices (tokens 0-7 | columns 0-7), (0-7 | 8-15), (8-15 | 0-7), (8-15 | 8-15)
        const uint32_t v_lane = smem_base + kSmemV + static_cast<uint32_t>((j4 >> 1) * 8 + r8) * 128u + static_cast<uint32_t>((2 * c + (j4 & 1)) ^ r8) * 16u;
        // blocks as B fragments: matrices (row half, column half) (0, 0), (0, 1), (1, 0), (1, 1); T^T transposed: (0, 0), (1, 0), (0, 1), (1, 1)
        const uint32_t b_lane = static_cast<uint32_t>((j4 & 1) * 256 + (j4 >> 1) * 128 + r8 * 16);
        const uint32_t l_lane = smem_base + kSmemL + b_lane, p_lane = smem_base + kSmemP + b_lane;
        const uint32_t t_lane = smem_base + kSmemL + static_cast<uint32_t>((j4 >> 1) * 256 + (j4 & 1) * 128 + r8 * 16);
        const float* alpha_sh = reinterpret_cast<const float*>(smem_gen + kSmemAlpha);
        uint32_t n = 0;
        for (unsigned u = blockIdx.x; u < total && ok; u += gridDim.x, ++n) {
            const uint32_t buf = n & 1u;
            ok = __all_sync(0xffffffffu, mbar_wait(bar_v + 8 * buf, (n >> 1) & 1u, 18));
            const uint32_t v_addr = v_lane + buf * kTileBytes;
            // The chain from one U to the next is two products; the sums over earlier blocks for the next X and for Y fill it.
            // Rows of L, T, P and the step sizes arrive and are given back 32 tokens at a time, so the next unit's follow while later rows of this one are
            // still read. (A wait that expires lets the unit run on, and the four warps agree behind it: its output stays unwritten, and all of them end their loop.)
            auto start_x = [&](int b, float (&X)[2][4]) {  // a V, transposed
                if (b % 2 == 0) ok = __all_sync(0xffffffffu, mbar_wait(bar_tri + 8 * (b / 2), n & 1u, 19)) && ok;
                uint32_t vf[4];
                ldmatrix_x4_trans(vf, v_addr + b * 2048);
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    const float2 al = *reinterpret_cast<const float2*>(alpha_sh + 16 * b + 8 * nt + 2 * tq);
                    const float2 lo = __fmul2_rn(al, __half22float2(*reinterpret_cast<const __half2*>(&vf[2 * nt])));
                    const float2 hi = __fmul2_rn(al, __half22float2(*reinterpret_cast<const __half2*>(&vf[2 * nt + 1])));
                    X[nt][0] = lo.x; X[nt][1] = lo.y; X[nt][2] = hi.x; X[nt][3] = hi.y;
                }
            };
            auto add = [&](float (&D)[2][4], const uint32_t (&A)[4], const uint32_t (&f)[4]) {
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) mma_f16_16816(D[nt], A[0], A[1], A[2], A[3], f[2 * nt], f[2 * nt + 1]);
            };
            auto packed = [&](const float (&D)[2][4], uint32_t (&A)[4]) {
                A[0] = pack_half2(D[0][0], D[0][1]);
                A[1] = pack_half2(D[0][2], D[0][3]);
                A[2] = pack_half2(D[1][0], D[1][1]);
                A[3] = pack_half2(D[1][2], D[1][3]);
            };
#pragma unroll
            for (int r = 0; r < R; ++r) {
                uint32_t U[NB][4];
                float X[2][4];
                start_x(r * NB, X);
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    const int b = r * NB + i;
                    if (b == 1 && n > 0 && warp == 4 && lane == 0) {  // the previous unit's output has left its buffer long ago
                        bulk_wait_read<0>();
                        mbar_arrive(bar_v_free + 8 * (buf ^ 1u));
                    }
                    uint32_t tf[4], f[4], x[4];
                    ldmatrix_x4_trans(tf, t_lane + tri(b, b));
                    if (i > 0) {
                        ldmatrix_x4(f, l_lane + tri(b, b - 1));
                        add(X, U[i - 1], f);
                    }
                    packed(X, x);
                    add(X, x, tf);  // U = X + (T - I) X: X itself is not rounded
                    float Xn[2][4], Y[2][4];
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) Xn[nt][e] = Y[nt][e] = 0.0f;
                    if (i + 1 < NB) start_x(b + 1, Xn);
#pragma unroll
                    for (int j = 0; j < i; ++j) {
                        if (i + 1 < NB) {
                            ldmatrix_x4(f, l_lane + tri(b + 1, r * NB + j));
                            add(Xn, U[j], f);
                        }
                        uint32_t pf[4];
                        ldmatrix_x4(pf, p_lane + tri(b, r * NB + j));
                        add(Y, U[j], pf);
                    }
                    ldmatrix_x4(f, p_lane + tri(b, b));
                    packed(X, U[i]);
                    add(Y, U[i], f);
                    stmatrix_x4_trans(v_addr + b * 2048, pack_half2(Y[0][0], Y[0][1]), pack_half2(Y[0][2], Y[0][3]), pack_half2(Y[1][0], Y[1][1]), pack_half2(Y[1][2], Y[1][3]));
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e) X[nt][e] = Xn[nt][e];
                    if (b % 2 == 1 || b == kUsed - 1) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_tri_free + 8 * (b / 2));
                    }
                }
            }
            fence_async_smem();
            ok = all_of_barrier1(ok);
            if (ok && warp == 4 && lane == 0) {
                const unsigned su = u / heads;
                const int seq = static_cast<int>(su * R), x = static_cast<int>(u - su * heads) * 64;
                tma_store_3d(&map_o, smem_base + kSmemV + buf * kTileBytes, x, 0, seq);  // (clips at T and at the last sequence)
                bulk_commit();
            }
        }
        if (warp == 4 && lane == 0) bulk_wait_read<0>();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

}  // namespace

// From 33 tokens on: up to 32 the chunked kernel's one or two chunks are as quick (one unit of 16 or 32 tokens 4.4 us there, 5.5 here). Never by the number of
// units: a sequence's bits do not depend on its company.
bool efla_tc_applies(const EflaParams& p) {
    return p.variant == BNF4_EFLA_AUTO && p.method == 1 && p.qkv_f16 && p.out_f16 && p.T > 32 && p.T <= kTok;
}

template <int NB>
static int launch_nb(const EflaParams& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mo, bool early, int dev, int sms, cudaStream_t stream) {
    static bool configured[64] = {};
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        const int rc = check_cuda(cudaFuncSetAttribute(efla_tc_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemAlloc), "cudaFuncSetAttribute(efla_tc_kernel)");
        if (rc) return rc;
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    const long long units = (p.seqs + kBlocks / NB - 1) / (kBlocks / NB) * p.heads;
    launch_pdl_if(early, efla_tc_kernel<NB>, static_cast<unsigned>(std::min<long long>(units, 2LL * sms)), kThreads, kSmemAlloc, stream, mq, mk, mv, mo, p);
    return check_launch("efla_tc_kernel");
}

int efla_tc_launch(const EflaParams& p, bool early, int dev, int sms, cudaStream_t stream) {
    const int nb = (p.T + 15) / 16;
    CUtensorMap mq, mk, mv, mo;
    auto map = [&](CUtensorMap* m, const void* base, int ld, const char* what) {
        return make_map_3d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, base, static_cast<uint64_t>(p.hidden), static_cast<uint64_t>(p.T), static_cast<uint64_t>(p.seqs),
                           static_cast<uint64_t>(ld) * 2, static_cast<uint64_t>(ld) * 2 * p.T, 64, 16 * nb, kBlocks / nb, what);
    };
    int rc = map(&mq, p.q, p.ld_qkv, "q");
    if (!rc) rc = map(&mk, p.k, p.ld_qkv, "k");
    if (!rc) rc = map(&mv, p.v, p.ld_qkv, "v");
    if (!rc) rc = map(&mo, p.out, p.ld_out, "scan output");
    if (rc) return rc;
    switch (nb) {
        case 3: return launch_nb<3>(p, mq, mk, mv, mo, early, dev, sms, stream);
        case 4: return launch_nb<4>(p, mq, mk, mv, mo, early, dev, sms, stream);
        case 5: return launch_nb<5>(p, mq, mk, mv, mo, early, dev, sms, stream);
        case 6: return launch_nb<6>(p, mq, mk, mv, mo, early, dev, sms, stream);
        case 7: return launch_nb<7>(p, mq, mk, mv, mo, early, dev, sms, stream);
        default: return launch_nb<8>(p, mq, mk, mv, mo, early, dev, sms, stream);
    }
}

int efla_tc_device_error(int* code) { return take_wait_error(code); }

}  // namespace bnf4
