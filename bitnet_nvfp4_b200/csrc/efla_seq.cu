// EFLA / DeltaNet recurrence of a whole sequence as dense contractions, for heads of any width: up to 128 tokens in one block, longer ones in
// blocks of 128 (efla_long_kernel).
//
// With a zero initial state the recurrence of efla.cu has a closed form that never builds the hd x hd state. Let
// k_t = n_t k^_t (n_t = |k_t|), w_t = alpha_t n_t (v_t - n_t k^_t . S_{t-1}), so that S_t = S_{t-1} + k^_t w_t^T. Then
//     (I + diag(a) strict(G)) w = diag(b) v,   G = K^ K^^T,  a_t = alpha_t n_t^2,  b_t = alpha_t n_t
//     y = P~ v,   P~ = lower(Q^ K^^T) (I + diag(a) strict(G))^-1 diag(b)
// P~ is a T x T lower-triangular matrix shared by all columns of the head, so one CTA per (sequence, head) computes it once and
// multiplies it with V: 2 T^2 hd multiply-adds per sequence instead of the 3 T hd^2 of the state form (six times fewer at
// T = 128, hd = 512), every input read once, no state, no scratch.
//
// Precision: every operand is split into two fp16 terms (x = hi + mid, 22 significant bits; rows of q and k are scaled by powers of
// two first, to a norm of 2^6 or more and values below 2^15, so that neither term under- or overflows) and the products hi hi + hi mid + mid hi accumulate in fp32. Nothing is
// rounded to fp16 between tokens, so the result lies closer to exact arithmetic than the per-token form's fp16 state.
//
// Values that are no numbers stay where the recurrence has them, although 0 x NaN is NaN in a contraction: from the first token on whose k or beta
// makes the state NaN, the sequence is cut off (as if it ended there) and the rows behind it are NaN; a v that is no number is taken out
// and its column is NaN from its token on; in q it only meets its own row.
//
// One CTA per (sequence, head), two or four where units leave SMs idle (each does steps 1 to 4 and a share of step 5); sixteen warps that work, one that issues the
// products, one that loads:
//   1. G and X = Q^ K^^T over 32-column blocks of K and Q: TMA into four slots, two groups of eight warps convert blocks in turn (fp32 -> two halves, rows scaled by powers of
//      two, squared norms on the way), six tcgen05 products of 128 x 128 per 16 columns accumulate in tensor memory, where the left operands lie too,
//   2. the per-token scalars; 1 / |q| and 1 / |k| reach G and X when they are read,
//   3. L and X into shared memory, inverses of the 16 x 16 diagonal blocks of I + L, L = diag(a) strict(G), by forward substitution in fp32,
//   4. P~ by block back substitution from the right with mma.sync, one warp per 16-row block (rows are independent, no barriers), into tensor memory,
//   5. y = P~ V over 64-column tiles of V (tcgen05, V's columns contiguous): eight warps convert tiles while the other eight take finished ones.
// No sum depends on which units share a launch.
// What bounds it: DRAM in steps 1 and 5 (29 and 26 k of 66 k cycles for a unit of 128 x 512; its input and output alone are 45 k of an SM's share), the chain of steps 3 and 4 in
// between. 1024 sequences of 128 tokens, one head of 512: 277 us; 32 sequences 27, of 16 tokens 18. The way there from 436 us: q and k read once and not for their norms
// first, loads that need no L1 lines (behind 200 KB of shared memory 28 KB of L1 held 60 % of the loads back) 436 -> 318; groups of eight warps instead of barriers of sixteen
// 318 -> 305; left operands in tensor memory 305 -> 277. Prefetches of the next unit into L2 (cp.async.bulk.prefetch, 11 bytes a cycle and SM) cost more than they hide.

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "mma_sync.cuh"
#include "tcgen05.cuh"

namespace bnf4 {

namespace {

// How the output lies to q, k or v: apart from it (also in other columns of the same rows), exactly in its place, in the same rows and by less than its width to
// the right, or in some other way.
enum SeqOverlap { SEQ_APART, SEQ_SAME, SEQ_RIGHT, SEQ_ACROSS };

constexpr int kSeqMaxT = 128;
constexpr int kSeqThreads = 512;
constexpr int kSqThreads = kSeqThreads + 64;       // efla_seq_kernel: sixteen warps that work, one that issues the products of steps 1 and 5, one the loads
constexpr int kSqStride = 72;                      // halves per row of the K / Q / V blocks: conflict-free ldmatrix rows
constexpr int kSqTile = kSeqMaxT * kSqStride * 2;  // bytes of one 128 x 64 block of halves
constexpr int kSqLStride = 136;                    // halves per row of L hi / L mid
constexpr int kSqXStride = 140;                    // floats per row of X (efla_seq_kernel), whose blocks P~'s replace; of the matrix of efla_long_kernel, P~ hi and mid
constexpr int kSqPMid = 272;                       // byte offset of P~ mid inside a row of the latter
constexpr int kSqTStride = 24;                     // halves per row of a diagonal block's inverse
// Shared memory of efla_seq_kernel. Step 1: K hi and K mid (64 columns, two halves of 32 in turn), behind them four slots of 32 columns of K and Q as they come
// from memory. Steps 3 and 4: L, X, the diagonal blocks and their inverses. Step 5: V hi and mid of two tiles, a finished tile of y, the odd tiles of V as they come. The even ones,
// the first of them from the start, have a place of their own.
constexpr int kSqUTile = kSeqMaxT * 128;                         // an operand tile: 128 rows x 64 halves, or 32 floats, 128B swizzle
constexpr int kSqRaw = 2 * kSqUTile;
constexpr int kSqX = 2 * kSeqMaxT * kSqLStride * 2;
constexpr int kSqDiag = kSqX + kSeqMaxT * kSqXStride * 4;        // fp32 diagonal blocks of L [8][16][17]
constexpr int kSqInv = kSqDiag + 8 * 16 * 17 * 4;                // their inverses, hi and mid [2][8][16][kSqTStride]
constexpr int kSqOut = 4 * kSqUTile;                             // 128 rows of 64 floats
constexpr int kSqV1 = 8 * kSqUTile, kSqV0 = 10 * kSqUTile;       // tiles of V: odd, even
constexpr int kSqScal = 12 * kSqUTile;                           // q factor, k factor, a, b [4][128] floats (first: largest values of the first columns)
constexpr int kSqScale = kSqScal + 4 * kSeqMaxT * 4;             // powers of two that scale the rows of q and k [2][128] floats
constexpr int kSqRed = kSqScale + 2 * kSeqMaxT * 4;              // reduction scratch [2][8], factors of two tiles of y, bad tokens [4]
constexpr int kSqPart = kSqRed + 256;                            // squared norms of q and k, four shares [4][2][128] floats
constexpr int kSqBad = kSqPart + 8 * kSeqMaxT * 4;               // first token of each of a tile's 64 columns whose v is no number, two tiles
constexpr int kSqBar = kSqBad + 2 * 64 * 4;                      // mbarriers, tensor memory slot
constexpr int kSqSmem = kSqBar + 256 + 1024;                     // (and room to align the tiles)
static_assert(kSqRaw + 8 * kSqUTile <= kSqV0 && kSqInv + 2 * 8 * 16 * kSqTStride * 2 <= kSqV0 && kSqSmem <= 232448, "regions");
// Tensor memory: G | X, then two tiles of y; behind them the left operands, which reach the products from here (from shared memory their reads, 4 KB for 64 cycles
// like the right operands', took step 1 to the limit of its bandwidth): K hi, K mid, Q hi, Q mid of two halves, then P~ hi and mid.
constexpr int kSqTmemCols = 512;
constexpr int kSqTA = 256;
constexpr uint32_t kSqIdesc = (1u << 4) | (static_cast<uint32_t>(kSeqMaxT >> 4) << 24);                        // fp16 x fp16 -> fp32, M 128
constexpr uint32_t kSqIdescY = kSqIdesc | (1u << 16) | (64u >> 3 << 17);  // N 64, B with columns contiguous
static_assert(kSqX % 16 == 0 && kSqDiag % 16 == 0 && kSqInv % 16 == 0 && kSqScal % 16 == 0, "16-byte aligned regions");
constexpr float kSqUp = 256.0f;                    // power-of-two scale of every normalised operand

// x0, x1 -> packed (hi, hi) and (mid, mid) halves with x = hi + mid to 22 bits
__device__ __forceinline__ void sq_split(float x0, float x1, uint32_t& hi, uint32_t& mid) {
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 hf = __half22float2(h);
    const __half2 m = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    mid = *reinterpret_cast<const uint32_t*>(&m);
}
// largest power of two that keeps |x| <= m below 2^TOP (1 for m == 0). V takes the most of fp16's range (TOP 15): its tokens share a scale, and what is
// 2^d below the largest of them keeps 22 bits up to d = 17 and 39 - d beyond. With 2^8 rows a factor of 1e7 smaller than later ones of
// their tile were off by 4e-3, more than fp16 states cost them.
template <int TOP>
__device__ __forceinline__ float sq_pow2_scale(float m) {
    if (!(m > 0.0f)) return 1.0f;
    const int e = static_cast<int>((__float_as_uint(m) >> 23) & 0xffu) - 127;  // 2^e <= m < 2^(e+1)
    return __uint_as_float(static_cast<uint32_t>(min(max(TOP - 1 - e + 127, 1), 254)) << 23);
}

// beta's logit and the squared norms of a token -> 1 / |q|, 1 / |k|, a and b
__device__ __forceinline__ void seq_scalars(const EflaParams& p, float logit, float qss, float kss, float& qinv, float& kinv, float& a, float& b) {
    const float beta = 1.0f / (1.0f + expf(-logit));
    const float lambda = kss < p.eps ? p.eps : kss;
    qinv = rsqrtf(qss + p.eps);
    kinv = kss > 0.0f ? rsqrtf(kss) : 0.0f;
    const float n = kss * kinv;
    const float ksc = p.method == 0 ? rsqrtf(lambda + p.eps) : 1.0f;
    const float alpha = p.method == 0 ? beta : -expm1f(-(beta * lambda)) / (lambda + p.eps);
    if (kss == INFINITY) {  // the norm of a finite k overflows: the recurrence leaves the state alone
        a = b = alpha * (p.method == 0 ? ksc : 1.0f);
    } else if (p.method == 0) {
        a = beta * (n * ksc) * (n * ksc);
        b = beta * (n * ksc);
    } else {
        a = alpha * kss;
        b = alpha * n;
    }
}
// The squared norm of a row (a warp's lanes hold its sum): infinite because of an infinite element (NaN then) or of an overflow?
__device__ __forceinline__ float seq_infinite_norm(float kss, const float* row, int hd, int lane) {
    if (kss != INFINITY) return kss;
    bool bad = false;
    for (int i = lane; i < hd; i += 32) bad = bad || !(fabsf(row[i]) <= FLT_MAX);
    return __any_sync(0xffffffffu, bad) ? NAN : kss;
}
// (one thread)
__device__ __forceinline__ float seq_infinite_norm(float kss, const float* row, int hd) {
    if (kss != INFINITY) return kss;
    for (int i = 0; i < hd; ++i)
        if (!(fabsf(row[i]) <= FLT_MAX)) return NAN;
    return kss;
}
__device__ __forceinline__ uint32_t seq_abs_bits(const float4& x) {  // ordered like the magnitudes, infinities and NaN above all numbers
    const uint32_t m = 0x7fffffffu;
    return max(max(__float_as_uint(x.x) & m, __float_as_uint(x.y) & m), max(__float_as_uint(x.z) & m, __float_as_uint(x.w) & m));
}
constexpr uint32_t kSeqNonFinite = 0x7f800000u;

// inverses of I + (diagonal 16 x 16 blocks of L): lane c owns column c of a block, two blocks per warp, four warps. Two halves, scaled by kSqUp.
__device__ __forceinline__ void seq_invert_diagonal(const float* Ld, __half* inv, int nb, int warp, int lane) {
    if (warp < 4) {
        const int blk = 2 * warp + (lane >> 4), c = lane & 15;
        if (blk < nb) {
            const float* d = Ld + blk * 16 * 17;
            float col[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                float x = t == c ? 1.0f : 0.0f;
#pragma unroll
                for (int s = 0; s < 16; ++s)
                    if (s < t) x = fmaf(-d[t * 17 + s], col[s], x);
                col[t] = x;
            }
            __half* ih = inv + blk * 16 * kSqTStride + c;
            __half* im = ih + 8 * 16 * kSqTStride;
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const float x = col[t] * kSqUp;
                const __half hi = __float2half_rn(x);
                ih[t * kSqTStride] = hi;
                im[t * kSqTStride] = __float2half_rn(x - __half2float(hi));
            }
        }
    }
}

// One warp: rows 16 i .. 16 i + 15 of P with P (I + L) = X by block columns from the right; L (two halves) at the start of
// shared memory, the diagonal blocks' inverses at inv_off; P (two halves, scaled by kSqUp) at mat_off (prow: the same place).
// X comes from get_x(j, n, e). PSTEP, PMID: bytes from a block's halves to the next block's, and to its mid halves.
template <int PSTEP, int PMID, class GetX>
__device__ __forceinline__ void seq_solve_rows(uint32_t sm0, uint32_t mat_off, uint8_t* prow, uint32_t inv_off, int i, int lane, GetX get_x) {
    const int g = lane >> 2, tq = lane & 3;
    const uint32_t p_addr = sm0 + mat_off + static_cast<uint32_t>((i * 16 + (lane & 15)) * (kSqXStride * 4) + (lane >> 4) * 16);
    const uint32_t l_addr = sm0 + static_cast<uint32_t>(((lane >> 3 & 1) * 8 + (lane & 7)) * kSqLStride + (lane >> 4) * 8) * 2u;
    const uint32_t i_addr = sm0 + inv_off + static_cast<uint32_t>(((lane >> 3 & 1) * 8 + (lane & 7)) * kSqTStride + (lane >> 4) * 8) * 2u;
    constexpr uint32_t kLMid = kSeqMaxT * kSqLStride * 2, kIMid = 8 * 16 * kSqTStride * 2;
    const float down = 1.0f / (kSqUp * kSqUp);
#pragma unroll
    for (int j = 7; j >= 0; --j) {
        if (j > i) continue;
        float s[2][4], c[2][4];  // sum over k > j of P~_ik L_kj: the large products and the cross terms in two chains
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = c[n][e] = 0.0f;
        for (int k = j + 1; k <= i; ++k) {
            uint32_t ph[4], pm[4], lh[4], lm[4];
            ldmatrix_x4(ph, p_addr + k * PSTEP);
            ldmatrix_x4(pm, p_addr + PMID + k * PSTEP);
            ldmatrix_x4_trans(lh, l_addr + k * (16 * kSqLStride * 2) + j * 32);
            ldmatrix_x4_trans(lm, l_addr + kLMid + k * (16 * kSqLStride * 2) + j * 32);
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                mma_f16_16816(s[n], ph, lh[2 * n], lh[2 * n + 1]);
                mma_f16_16816(c[n], ph, lm[2 * n], lm[2 * n + 1]);
                mma_f16_16816(c[n], pm, lh[2 * n], lh[2 * n + 1]);
            }
        }
        // z = X_ij - sum, then P~_ij = z inv_jj
        uint32_t zh[4], zm[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            float z[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) z[e] = (get_x(j, n, e) - (s[n][e] + c[n][e]) * down) * kSqUp;
            sq_split(z[0], z[1], zh[2 * n], zm[2 * n]);
            sq_split(z[2], z[3], zh[2 * n + 1], zm[2 * n + 1]);
        }
        uint32_t th[4], tm[4];
        ldmatrix_x4_trans(th, i_addr + j * (16 * kSqTStride * 2));
        ldmatrix_x4_trans(tm, i_addr + kIMid + j * (16 * kSqTStride * 2));
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            float o[4] = {0.0f, 0.0f, 0.0f, 0.0f}, oc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_f16_16816(o, zh, th[2 * n], th[2 * n + 1]);
            mma_f16_16816(oc, zh, tm[2 * n], tm[2 * n + 1]);
            mma_f16_16816(oc, zm, th[2 * n], th[2 * n + 1]);
            const int c0 = j * PSTEP + (n * 8 + 2 * tq) * 2;
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                uint32_t hi, mid;
                sq_split((o[2 * hr] + oc[2 * hr]) * (1.0f / kSqUp), (o[2 * hr + 1] + oc[2 * hr + 1]) * (1.0f / kSqUp), hi, mid);
                uint8_t* d = prow + (i * 16 + g + 8 * hr) * (kSqXStride * 4) + c0;
                *reinterpret_cast<uint32_t*>(d) = hi;
                *reinterpret_cast<uint32_t*>(d + PMID) = mid;
            }
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void sq_tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
                 "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void sq_tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// A from tensor memory: lane = row, two halves per column
__device__ __forceinline__ void sq_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void sq_tmem_ld16(uint32_t taddr, float (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]),
          "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
        : "r"(taddr)
        : "memory");
}

// The largest values of the rows of q and k [2][128], a warp (of sixteen) per row
__device__ __forceinline__ void seq_row_maxima(const float* qg, const float* kg, int ld, int T, int hd, float* out) {
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x >> 5; t < T; t += kSeqThreads / 32) {
        float m[2] = {0.0f, 0.0f};
        const float *qr = qg + static_cast<size_t>(t) * ld, *kr = kg + static_cast<size_t>(t) * ld;
#pragma unroll 4
        for (int c = 4 * lane; c < hd; c += 128) {
            const float4 x = *reinterpret_cast<const float4*>(qr + c), y = *reinterpret_cast<const float4*>(kr + c);
            m[0] = fmaxf(m[0], fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
            m[1] = fmaxf(m[1], fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w))));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(m[i]));
            if (lane == 0) out[i * kSeqMaxT + t] = __uint_as_float(bits);
        }
    }
}

// cs CTAs share a unit: each does steps 1 to 4 (the same sums) and its share of the column tiles of step 5. meet: they form a cluster, and none writes
// before all have read q and k, where the output may lie. across: it may lie on v, on other columns (SeqOverlap).
__global__ void __launch_bounds__(kSqThreads, 1) efla_seq_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                                                                 const __grid_constant__ CUtensorMap map_v, const EflaParams p, const int cs, const int meet, const int across) {
    pdl_wait();
    extern __shared__ uint8_t sm_raw[];
    uint8_t* sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);
    const uint32_t sm0 = smem_u32(sm);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = p.T, hd = p.hidden / p.heads;
    const unsigned unit = blockIdx.x / static_cast<unsigned>(cs);
    const int nd = (hd + 63) >> 6;  // 64-column blocks
    const int share = static_cast<int>(blockIdx.x - unit * static_cast<unsigned>(cs));
    const int ct0 = share * nd / cs, nct = (share + 1) * nd / cs - ct0;  // this CTA's column tiles of y
    const unsigned seq = unit / static_cast<unsigned>(p.heads);
    const int h = static_cast<int>(unit - seq * static_cast<unsigned>(p.heads));
    const int nb = (T + 15) >> 4;  // 16-token blocks: nothing behind them is converted or multiplied
    const size_t row0 = static_cast<size_t>(seq) * T;
    const float* qg = static_cast<const float*>(p.q) + row0 * p.ld_qkv + h * hd;
    const float* kg = static_cast<const float*>(p.k) + row0 * p.ld_qkv + h * hd;
    const float* vg = static_cast<const float*>(p.v) + row0 * p.ld_qkv + h * hd;
    float* og = static_cast<float*>(p.out) + row0 * p.ld_out + h * hd;

    float* qs_sh = reinterpret_cast<float*>(sm + kSqScal);
    float* ks_sh = qs_sh + kSeqMaxT;
    float* a_sh = ks_sh + kSeqMaxT;
    float* b_sh = a_sh + kSeqMaxT;
    float* red = reinterpret_cast<float*>(sm + kSqRed);
    int* red_bad = reinterpret_cast<int*>(red + 48);  // [4]
    volatile int* stop = reinterpret_cast<volatile int*>(red + 52);
    float* part = reinterpret_cast<float*>(sm + kSqPart);
    // mbarriers: slots of K and Q filled / read (four each), halves of the operands complete / multiplied (two each), tiles of V filled / read (two each), operands of V
    // complete, tiles of y complete / read (two each)
    const uint32_t bar0 = sm0 + kSqBar, bar_raw = bar0, bar_read = bar0 + 32, bar_op = bar0 + 64, bar_mul = bar0 + 80, bar_v = bar0 + 96, bar_vread = bar0 + 112, bar_vop = bar0 + 128, bar_y = bar0 + 144,
                   bar_drain = bar0 + 160;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + kSqBar + 192);
    constexpr int kGroup = kSeqThreads / 64;  // warps of one of the two groups that share steps 1 and 5
    if (tid == 0) {
        *stop = 0;
        for (int b = 0; b < 4; ++b) { mbar_init(bar_raw + 8 * b, 1); mbar_init(bar_read + 8 * b, kGroup); }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_op + 8 * b, kGroup);
            mbar_init(bar_mul + 8 * b, 1);
            mbar_init(bar_v + 8 * b, 1);
            mbar_init(bar_vread + 8 * b, kGroup);
            mbar_init(bar_vop + 8 * b, kGroup);
            mbar_init(bar_y + 8 * b, 1);
            mbar_init(bar_drain + 8 * b, kGroup);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 16) {
        tmem_alloc(bar0 + 192, kSqTmemCols);
        tmem_relinquish();
    }
    // No wait of this thread has expired; behind one that has there are no others. `stop` tells the other threads: what follows an expired wait, whichever warp's, may
    // rest on operands that never came, and stays unwritten. (It is set in front of the arrivals that lead there, and read behind them.)
    bool ok = true;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) {
        if (ok && !mbar_wait(bar, parity, code)) {
            ok = false;
            *stop = 1;
        }
    };

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // ---------------- 1. G and X of rows scaled by powers of two, squared norms on the way ----------------
    // 32 columns at a time: a warp loads (TMA), two groups of eight convert them in turn (thread = sixteen columns of a row of K and of Q), one issues the products.
    const int nh = hd >> 5, group = warp >> 3, quad = warp & 3, ch = (warp >> 2) & 1;
    const int t_row = 32 * quad + lane;  // this thread's row, and its lane of tensor memory
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(32 * quad) << 16);
    const int swz = t_row & 7;
    float* scale_sh = reinterpret_cast<float*>(sm + kSqScale);
    auto workers_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kSeqThreads) : "memory"); };
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(2 + group), "n"(kSeqThreads / 2) : "memory"); };
    const int x0 = h * hd, y0 = static_cast<int>(row0);
    auto put_split = [&](uint8_t* at, const float4& x, float s, int mid_off) {
        uint2 hi, mid;
        sq_split(x.x * s, x.y * s, hi.x, mid.x);
        sq_split(x.z * s, x.w * s, hi.y, mid.y);
        *reinterpret_cast<uint2*>(at) = hi;
        *reinterpret_cast<uint2*>(at + mid_off) = mid;
    };
    auto arrive = [&](uint32_t bar) {  // this warp's share of an operand is in shared memory
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
    };
    auto abs4 = [](const float4& x) { return fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))); };
    auto sumsq = [](float s, const float4& x) {
        s = fmaf(x.x, x.x, s); s = fmaf(x.y, x.y, s); s = fmaf(x.z, x.z, s);
        return fmaf(x.w, x.w, s);
    };
    // An output to the right of v is formed from the last column tile to the first: a tile then lies on columns that have been read, however far to the right.
    auto tile_col = [&](int l) { return (ct0 + (across == SEQ_RIGHT ? nct - 1 - l : l)) * 64; };
    const uint32_t box_bytes = static_cast<uint32_t>(T) * 128;  // the rows of one sequence; nothing is read behind them
    int v_loads = 0;
    auto load_v = [&](int l) {  // (the loading warp) the CTA's l-th tile of V: two boxes of 32 columns, or the one that is left
        const uint32_t at = sm0 + ((l & 1) ? kSqV1 : kSqV0);
        const int c = tile_col(l);
        if (elect_one()) {
            const bool two = c + 32 < hd;
            mbar_expect_tx(bar_v + 8 * (l & 1), (two ? 2 : 1) * box_bytes);
            tma_load_2d(at, &map_v, x0 + c, y0, bar_v + 8 * (l & 1));
            if (two) tma_load_2d(at + kSqUTile, &map_v, x0 + c + 32, y0, bar_v + 8 * (l & 1));
        }
        __syncwarp();
        ++v_loads;
    };
    // The scale of a row is taken from its first 32 columns (largest value just below 2^8), so that q and k are read once; a row that leaves the range of
    // halves later on, or has only zeros there, sends the whole unit through a second pass with scales from whole rows. One head of 512, a row of every unit being
    // such: 1024 x 128 tokens 277 -> 403 us, 32 x 128 26.4 -> 41.8, 1024 x 33 180 -> 249 (with a thread per row for the largest values 508, 56.7, 295). The passes are
    // two instances of one body: tests for the pass inside it cost 0.8 us of 17.9 at one token.
    auto norm2 = [&](int m, int t) { return (part[m * kSeqMaxT + t] + part[(2 + m) * kSeqMaxT + t]) + (part[(4 + m) * kSeqMaxT + t] + part[(6 + m) * kSeqMaxT + t]); };
    int loads = 0;  // blocks of K and Q that the loading warp has asked for
    auto step1 = [&](auto second) {  // does a row leave the range?
        constexpr bool kSecond = decltype(second)::value;
        const int it0 = kSecond ? nh : 0;  // blocks before this pass: the barriers' phases go on
        if (warp < 16) {
            float ss[2] = {0.0f, 0.0f}, sc[2];  // k, q
            for (int hb = group; hb < nh; hb += 2) {
                const int it = it0 + hb, slot = it & 3, half = it & 1;
                wait(bar_raw + 8 * slot, static_cast<uint32_t>(it >> 2) & 1u, 26);
                const uint8_t* raw = sm + kSqRaw + slot * (2 * kSqUTile) + t_row * 128;
                float4 x[2][4];
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        x[m][j] = t_row < T ? *reinterpret_cast<const float4*>(raw + m * kSqUTile + (((4 * ch + j) ^ swz) << 4)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (hb == group) {  // the scales, from the first block: the largest values of its columns 16 ch ..
                    if (group == 0) {
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            float mx = fmaxf(fmaxf(abs4(x[m][0]), abs4(x[m][1])), fmaxf(abs4(x[m][2]), abs4(x[m][3])));
                            if (kSecond && t_row < T) mx = fmaxf(mx, scale_sh[(1 - m) * kSeqMaxT + t_row]);
                            qs_sh[(2 * m + ch) * kSeqMaxT + t_row] = mx;
                        }
                    }
                    workers_sync();
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        sc[m] = sq_pow2_scale<8>(fmaxf(qs_sh[2 * m * kSeqMaxT + t_row], qs_sh[(2 * m + 1) * kSeqMaxT + t_row]));
                        if (group == 0 && ch == 0) scale_sh[(1 - m) * kSeqMaxT + t_row] = sc[m];
                    }
                }
                if (it >= 2) wait(bar_mul + 8 * half, static_cast<uint32_t>(it / 2 - 1) & 1u, 21);  // the half's last products have read it
                __syncwarp();
                tc_fence_after();
                if (32 * quad < 16 * nb) {
                    const uint32_t ta = t_lane + kSqTA + 64 * half + 8 * ch;
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        uint32_t hi[8], mid[8];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 y = x[m][j];
                            ss[m] = sumsq(ss[m], y);
                            sq_split(y.x * sc[m], y.y * sc[m], hi[2 * j], mid[2 * j]);
                            sq_split(y.z * sc[m], y.w * sc[m], hi[2 * j + 1], mid[2 * j + 1]);
                        }
                        if (m == 0) {  // K is the right operand too
                            uint8_t* row = sm + t_row * 128;
#pragma unroll
                            for (int j = 0; j < 2; ++j) {
                                const int at = ((4 * half + 2 * ch + j) ^ swz) << 4;
                                *reinterpret_cast<uint4*>(row + at) = make_uint4(hi[4 * j], hi[4 * j + 1], hi[4 * j + 2], hi[4 * j + 3]);
                                *reinterpret_cast<uint4*>(row + kSqUTile + at) = make_uint4(mid[4 * j], mid[4 * j + 1], mid[4 * j + 2], mid[4 * j + 3]);
                            }
                        }
                        sq_tmem_st8(ta + 32 * m, hi);
                        sq_tmem_st8(ta + 32 * m + 16, mid);
                    }
                    sq_tmem_st_wait();
                }
                tc_fence_before();
                arrive(bar_op + 8 * half);
                if (lane == 0) mbar_arrive(bar_read + 8 * slot);  // (behind the stores of what was read: released behind the loads alone, the slot was filled again under them)
            }
            part[((2 * group + ch) * 2 + 1) * kSeqMaxT + t_row] = ss[0];
            part[(2 * group + ch) * 2 * kSeqMaxT + t_row] = ss[1];
        } else if (warp == 16) {
            // The products have a warp of their own: their issue waits for the tensor pipe (64 cycles each, 12 to a block), which held up the conversions
            // of the warp that did both, and with it every barrier.
            const uint64_t kh = smem_desc(sm0, 16, 1024, kLayoutSw128), km = smem_desc(sm0 + kSqUTile, 16, 1024, kLayoutSw128);
            const uint32_t gram = kSqIdesc | (static_cast<uint32_t>(2 * nb) << 17);  // N 16 nb
            for (int hb = 0; hb < nh; ++hb) {
                const int it = it0 + hb, half = it & 1;
                wait(bar_op + 8 * half, static_cast<uint32_t>(it / 2) & 1u, 24);
                if (elect_one() && ok) {
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk) {  // hi hi + hi mid + mid hi
                        const uint64_t o = static_cast<uint64_t>(4 * half + 2 * kk);
                        const uint32_t ta = tmem + kSqTA + 64 * half + 8 * kk, more = hb > 0 || kk > 0 ? 1u : 0u;
                        sq_mma_ts(tmem, ta, kh + o, gram, more);
                        sq_mma_ts(tmem + 128, ta + 32, kh + o, gram, more);
                        sq_mma_ts(tmem, ta, km + o, gram, 1u);
                        sq_mma_ts(tmem + 128, ta + 32, km + o, gram, 1u);
                        sq_mma_ts(tmem, ta + 16, kh + o, gram, 1u);
                        sq_mma_ts(tmem + 128, ta + 48, kh + o, gram, 1u);
                    }
                    tc_commit(bar_mul + 8 * half);
                }
                __syncwarp();
            }
        } else {
            for (int hb = 0; hb < nh; ++hb) {
                const int it = it0 + hb, slot = it & 3;
                if (it >= 4) wait(bar_read + 8 * slot, static_cast<uint32_t>(it / 4 - 1) & 1u, 27);
                if (!__all_sync(0xffffffffu, ok)) break;
                if (elect_one()) {
                    const uint32_t at = sm0 + kSqRaw + slot * (2 * kSqUTile);
                    mbar_expect_tx(bar_raw + 8 * slot, 2 * box_bytes);
                    tma_load_2d(at, &map_k, x0 + 32 * hb, y0, bar_raw + 8 * slot);
                    tma_load_2d(at + kSqUTile, &map_q, x0 + 32 * hb, y0, bar_raw + 8 * slot);
                }
                __syncwarp();
                ++loads;
                if (!kSecond && hb == min(3, nh - 1)) load_v(0);
            }
        }
        for (int it = max(0, it0 + nh - 2); it < it0 + nh; ++it) wait(bar_mul + 8 * (it & 1), static_cast<uint32_t>(it / 2) & 1u, 22);
        tc_fence_after();
        __syncthreads();  // (everyone has seen the products done before their operands' places are taken)
        bool again = false;
        if (!kSecond && tid < T) {
            // A scaled value may be beyond 2^15, or the row is below 2^6, where the mid halves run out of bits (first columns that are not zero make it 2^7 at least). Squares of
            // values below 2^-75 are lost: these stay below 2^15 under scales of up to 2^90.
            auto leaves = [](float sum, float s) {
                const float v = sum * s * s;
                return sum > 0.0f ? !(v >= 4096.0f && v <= 1073741824.0f) : s > 0x1p90f;
            };
            again = leaves(norm2(0, tid), scale_sh[tid]) || leaves(norm2(1, tid), scale_sh[kSeqMaxT + tid]);
        }
        return !kSecond && __syncthreads_or(again) != 0;
    };
    if (step1(std::false_type())) {
        if (warp < 16) {
            seq_row_maxima(qg, kg, p.ld_qkv, T, hd, scale_sh);
            workers_sync();
        }
        step1(std::true_type());
    }

    // ---------------- 2. scalars of the tokens ----------------
    if (tid < kSeqMaxT) {
        const int t = tid;
        float a = 0.0f, b = 0.0f, kinv = 0.0f, qinv = 0.0f;
        if (t < T) {
            const float bias = efla_seq_bias(p, static_cast<unsigned>(seq));
            seq_scalars(p, p.beta_raw[(row0 + t) * p.ld_beta] + bias, norm2(0, t), seq_infinite_norm(norm2(1, t), kg + static_cast<size_t>(t) * p.ld_qkv, hd), qinv, kinv, a, b);
        }
        qs_sh[t] = qinv / scale_sh[t];  // (powers of two: exact)
        ks_sh[t] = kinv / scale_sh[kSeqMaxT + t];
        a_sh[t] = a;
        b_sh[t] = b;
        float m = b;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const uint32_t bad = __reduce_min_sync(0xffffffffu, static_cast<uint32_t>(a == a && b == b ? T : t));
        if (lane == 0) { red[warp] = m; red_bad[warp] = static_cast<int>(bad); }
    }
    __syncthreads();
    const int Te = min(min(red_bad[0], red_bad[1]), min(red_bad[2], red_bad[3]));  // tokens before the first one that makes the state NaN
    if (Te < T) {
        if (tid >= Te && tid < T) a_sh[tid] = b_sh[tid] = 0.0f;
        __syncthreads();
    }
    const float bscale = sq_pow2_scale<6>(fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3])));  // b * bscale < 64: P~ below 2^14, also for V's sake
    if (meet) cluster_sync();
    // ---------------- 3. L (two halves), its diagonal blocks (fp32), X (fp32): a thread per row and 32 columns ----------------
    __half* Lh = reinterpret_cast<__half*>(sm);
    float* X = reinterpret_cast<float*>(sm + kSqX);
    float* Ld = reinterpret_cast<float*>(sm + kSqDiag);
    const int cg = warp >> 2;  // columns 32 cg ..
    if (cg <= quad && 32 * quad < 16 * nb) {  // (the seventeenth warp has no columns: cg 4)
        const bool row_ok = t_row < Te;  // (behind the cut there may be values that are no numbers)
        const float at = a_sh[t_row], gf = ks_sh[t_row], xf = qs_sh[t_row];
#pragma unroll
        for (int hc = 0; hc < 2; ++hc) {  // sixteen columns at a time
            const int c0 = 32 * cg + 16 * hc;
            if (c0 >= 16 * nb) break;
            float g[16], x[16];
            sq_tmem_ld16(t_lane + c0, g);
            sq_tmem_ld16(t_lane + 128 + c0, x);
            tmem_ld_wait();
            uint32_t hi[8], mid[8];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float f = ks_sh[c0 + e];
                g[e] = row_ok && c0 + e < t_row ? at * (g[e] * gf * f) : 0.0f;
                x[e] = row_ok && c0 + e <= t_row ? x[e] * xf * f : 0.0f;
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) sq_split(g[2 * e] * kSqUp, g[2 * e + 1] * kSqUp, hi[e], mid[e]);
            uint4* l = reinterpret_cast<uint4*>(Lh + t_row * kSqLStride + c0);
            uint4* lm = reinterpret_cast<uint4*>(Lh + (kSeqMaxT + t_row) * kSqLStride + c0);
            l[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            l[1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
            lm[0] = make_uint4(mid[0], mid[1], mid[2], mid[3]);
            lm[1] = make_uint4(mid[4], mid[5], mid[6], mid[7]);
            float4* xr = reinterpret_cast<float4*>(X + t_row * kSqXStride + c0);
#pragma unroll
            for (int e = 0; e < 4; ++e) xr[e] = make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
            if (c0 >> 4 == t_row >> 4) {
#pragma unroll
                for (int e = 0; e < 16; ++e) Ld[t_row * 17 + e] = g[e];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    // inverse of I + L_ii: lane c owns column c of a block, two blocks per warp
    seq_invert_diagonal(Ld, reinterpret_cast<__half*>(sm + kSqInv), nb, warp, lane);
    __syncthreads();

    // ---------------- 4. P~ M = X by block columns from the right; warp i owns rows 16 i .. 16 i + 15 ----------------
    const int g = lane >> 2, tq = lane & 3;
    uint8_t* prow = sm + kSqX;
    if (warp < nb) {
        // P~'s blocks, two halves a value, take the place of X's as they are finished (32 bytes a row each: hi, mid)
        const int i = warp;
        const float* xi = X + (i * 16 + g) * kSqXStride + 2 * tq;
        seq_solve_rows<64, 32>(sm0, kSqX, prow, kSqInv, i, lane, [&](int j, int n, int e) { return xi[(e >> 1) * 8 * kSqXStride + j * 16 + n * 8 + (e & 1)]; });
    }
    __syncthreads();  // P~ is complete
    if (warp < 16 && 32 * quad < 16 * nb) {
        // the columns' factors b_s, scaled to at most 64, applied to the finished rows (exact powers of two aside, one more rounding); zeros above the diagonal
        const uint32_t ta = t_lane + kSqTA;
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
            const int j = 2 * cg + jj;
            if (j >= nb) break;
            uint32_t hi[8], mid[8];
            const uint4* d = reinterpret_cast<const uint4*>(prow + t_row * (kSqXStride * 4) + j * 64);
            const float4* bs = reinterpret_cast<const float4*>(b_sh + 16 * j);
#pragma unroll
            for (int e = 0; e < 8; ++e) hi[e] = mid[e] = 0u;
            if (j <= t_row >> 4) {
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const uint4 hv = d[v], mv = d[2 + v];
                    const uint32_t hw[4] = {hv.x, hv.y, hv.z, hv.w}, mw[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&hw[e])), mf = __half22float2(*reinterpret_cast<const __half2*>(&mw[e]));
                        const float4 b4 = bs[2 * v + (e >> 1)];
                        const float b0 = (e & 1) ? b4.z : b4.x, b1 = (e & 1) ? b4.w : b4.y;
                        sq_split((hf.x + mf.x) * (b0 * bscale), (hf.y + mf.y) * (b1 * bscale), hi[4 * v + e], mid[4 * v + e]);
                    }
                }
            }
            __syncwarp();
            sq_tmem_st8(ta + 8 * j, hi);
            sq_tmem_st8(ta + 64 + 8 * j, mid);
        }
        sq_tmem_st_wait();
    }
    tc_fence_before();
    fence_async_smem();
    __syncthreads();  // (also: the rows of P~ have been read, V's tiles take their place)

    // ---------------- 5. y = P~ V, 64 columns at a time; a tile leaves while the next ones are converted and multiplied ----------------
    const bool wide = ((reinterpret_cast<uintptr_t>(p.out) & 15) | (p.ld_out & 3)) == 0;  // rows of y start at multiples of 16 bytes
    float* ds_sh = red + 16;                                  // [2]: undoes the scales of P~ and of V
    int* bad_sh = reinterpret_cast<int*>(red + 18);           // [2]: a v of the tile is no number
    if (warp < kGroup) {
        // eight warps convert V (thread = a 16-byte piece of eight rows) ..
        const int piece = tid & 15, srow = tid >> 4;
        constexpr int kRows = kSeqThreads / 32, kPer = kSeqMaxT / kRows;
        for (int l = 0; l < nct; ++l) {
            float4 v[kPer];
            wait(bar_v + 8 * (l & 1), static_cast<uint32_t>(l / 2) & 1u, 28);
            const int c = tile_col(l) + 4 * piece;
            const uint8_t* raw = sm + ((l & 1) ? kSqV1 : kSqV0) + (piece >> 3) * kSqUTile + srow * 128 + (((piece & 7) ^ (srow & 7)) << 4);
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                v[i] = srow + kRows * i < Te && c < hd ? *reinterpret_cast<const float4*>(raw + i * (kRows * 128)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            // the tile's own power-of-two scale keeps both halves of its values in range
            uint32_t m = 0;
#pragma unroll
            for (int i = 0; i < kPer; ++i) m = max(m, seq_abs_bits(v[i]));
            m = __reduce_max_sync(0xffffffffu, m);
            uint32_t* redb = reinterpret_cast<uint32_t*>(red) + 8 * (l & 1);
            if (lane == 0) {
                redb[warp] = m;
                mbar_arrive(bar_vread + 8 * (l & 1));  // (the tile has been read: its values are in m)
            }
            if (l >= 2) wait(bar_drain + 8 * (l & 1), static_cast<uint32_t>(l / 2 - 1) & 1u, 27);  // the tile before the last has left its accumulator (and its product the operands)
            group_sync();
            m = __reduce_max_sync(0xffffffffu, redb[lane & 7]);
            const bool tile_bad = m >= kSeqNonFinite;
            if (tile_bad) {
                int* bad_col = reinterpret_cast<int*>(sm + kSqBad) + 64 * (l & 1);
                if (tid < 64) bad_col[tid] = T;
                group_sync();
                m = 0;
#pragma unroll
                for (int i = 0; i < kPer; ++i) {
                    auto clear = [&](float& x, int e) {
                        if (!(fabsf(x) <= FLT_MAX)) {
                            atomicMin(bad_col + 4 * piece + e, srow + kRows * i);
                            x = 0.0f;
                        }
                    };
                    clear(v[i].x, 0); clear(v[i].y, 1); clear(v[i].z, 2); clear(v[i].w, 3);
                    m = max(m, seq_abs_bits(v[i]));
                }
                m = __reduce_max_sync(0xffffffffu, m);
                if (lane == 0) redb[warp] = m;  // (read by everyone before the barrier above)
                group_sync();
                m = __reduce_max_sync(0xffffffffu, redb[lane & 7]);
            }
            const float vs = sq_pow2_scale<15>(__uint_as_float(m));
            if (tid == 0) {
                ds_sh[l & 1] = 1.0f / kSqUp / bscale / vs;  // (P~'s scales are 2^8 and b's)
                bad_sh[l & 1] = tile_bad;
            }
            uint8_t* st = sm + (l & 1) * (2 * kSqUTile) + srow * 128 + (((piece >> 1) ^ (srow & 7)) << 4) + (piece & 1) * 8;
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                if (srow + kRows * i < 16 * nb) put_split(st + i * (kRows * 128), v[i], vs, kSqUTile);
            arrive(bar_vop + 8 * (l & 1));
        }
    } else if (warp < 16) {
        // .. and eight take the tiles of y: rows t of 256 bytes, 16-byte piece ^ t % 16: a row's 32 columns go in, whole rows of the output come out, both without bank conflicts
        float* out = reinterpret_cast<float*>(sm + kSqOut);
        const int half = ch, gtid = tid - 32 * kGroup;
        for (int l = 0; l < nct; ++l) {
            wait(bar_vop + 8 * (l & 1), static_cast<uint32_t>(l / 2) & 1u, 29);
            const float ds = ds_sh[l & 1];
            const bool tile_bad = bad_sh[l & 1] != 0;
            wait(bar_y + 8 * (l & 1), static_cast<uint32_t>(l / 2) & 1u, 23);
            __syncwarp();
            tc_fence_after();
            uint32_t acc[32];
            tmem_ld32(t_lane + (l & 1) * 64 + 32 * half, acc);
            tmem_ld_wait();
            tc_fence_before();
            float y[32];
            const int* bad_col = reinterpret_cast<const int*>(sm + kSqBad) + 64 * (l & 1);
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                y[e] = __uint_as_float(acc[e]) * ds;
                if (tile_bad || Te < T)
                    if (t_row >= Te || (tile_bad && t_row >= bad_col[32 * half + e])) y[e] = NAN;
            }
            if (l > 0) group_sync();  // the tile before has left `out`
#pragma unroll
            for (int e = 0; e < 8; ++e)
                *reinterpret_cast<float4*>(out + t_row * 64 + (((8 * half + e) ^ (t_row & 15)) << 2)) = make_float4(y[4 * e], y[4 * e + 1], y[4 * e + 2], y[4 * e + 3]);
            // SEQ_ACROSS: y may lie on other columns of v and leaves when the next three tiles have been read or are here. The last of them is waited for in front of this
            // arrival: without it no warp reads that tile, so that the copy after next, which would complete the same barrier once more, cannot pass the wait.
            if (across == SEQ_ACROSS && l + 3 < nct) wait(bar_v + 8 * ((l + 3) & 1), static_cast<uint32_t>((l + 3) / 2) & 1u, 28);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_drain + 8 * (l & 1));
            if (across == SEQ_ACROSS && l + 2 < nct) wait(bar_vop + 8 * (l & 1), static_cast<uint32_t>(l / 2 + 1) & 1u, 29);
            group_sync();
            const bool write = *stop == 0;  // (no way out of the loop: threads that read it before and after it is set would part at the barriers)
            if (wide) {
                const int piece = gtid & 15, c = tile_col(l) + 4 * piece;
#pragma unroll 4
                for (int t = gtid >> 4; t < T; t += kSeqThreads / 32)
                    if (write && c < hd) *reinterpret_cast<float4*>(og + static_cast<size_t>(t) * p.ld_out + c) = *reinterpret_cast<const float4*>(out + t * 64 + ((piece ^ (t & 15)) << 2));
            } else {
                const int c = tile_col(l) + 2 * lane;
                for (int t = warp - kGroup; t < T; t += kGroup)
                    if (write && c < hd) *reinterpret_cast<float2*>(og + static_cast<size_t>(t) * p.ld_out + c) = *reinterpret_cast<const float2*>(out + t * 64 + (((lane >> 1) ^ (t & 15)) << 2) + 2 * (lane & 1));
            }
        }
    } else if (warp == 16) {
        for (int l = 0; l < nct; ++l) {
            wait(bar_vop + 8 * (l & 1), static_cast<uint32_t>(l / 2) & 1u, 25);
            if (elect_one() && ok) {
                tc_fence_after();
                const uint32_t at = sm0 + (l & 1) * (2 * kSqUTile), d = tmem + (l & 1) * 64, ta = tmem + kSqTA;
                const uint64_t vh = smem_desc(at, 1024, 1024, kLayoutSw128), vm = smem_desc(at + kSqUTile, 1024, 1024, kLayoutSw128);
                for (int kk = 0; kk < nb; ++kk) {  // sixteen tokens: 8 columns of P~, 16 rows of V
                    const uint64_t b = static_cast<uint64_t>(kk * (2048 >> 4));
                    sq_mma_ts(d, ta + 8 * kk, vh + b, kSqIdescY, kk > 0 ? 1u : 0u);
                    sq_mma_ts(d, ta + 8 * kk, vm + b, kSqIdescY, 1u);
                    sq_mma_ts(d, ta + 64 + 8 * kk, vh + b, kSqIdescY, 1u);
                }
                tc_commit(bar_y + 8 * (l & 1));
            }
            __syncwarp();
        }
    } else {
        for (int l = 1; l < nct; ++l) {
            if (l >= 2) wait(bar_vread + 8 * (l & 1), static_cast<uint32_t>(l / 2 - 1) & 1u, 29);
            if (!__all_sync(0xffffffffu, ok)) break;
            load_v(l);
        }
        // none of the copies may be on its way when the CTA leaves (they have all been waited for unless a wait expired)
        for (int s = 0; s < 4; ++s)
            if (loads > s) mbar_wait(bar_raw + 8 * s, static_cast<uint32_t>((loads - 1 - s) / 4) & 1u, 26);
        for (int s = 0; s < 2; ++s)
            if (v_loads > s) mbar_wait(bar_v + 8 * s, static_cast<uint32_t>((v_loads - 1 - s) / 2) & 1u, 28);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        tmem_dealloc(tmem, kSqTmemCols);
    }
}

// ------------------------------------------------------------------------------------------------
// The same closed form for sequences of more than 128 tokens, one CTA per (sequence, head), 128-token blocks. With r_I = diag(b) v_I -
// sum_{J < I} L_IJ w_J the blocks of w = (I + L)^-1 diag(b) v follow one after the other, w_I = (I + L_II)^-1 r_I, and y_I = sum_{J <= I} X_IJ w_J.
// w lives in the rows of the output until its block's y replaces it: blocks of y are formed from the last to the first, and y_I needs w_J of
// J <= I only, so there is no scratch. Every block product goes through one gram routine (two blocks of rows over hd -> 128 x 128
// matrix in shared memory, two halves per element) and one product routine (that matrix times a 128 x hd block, 64 columns at a time).
// T^2 hd products on the tensor cores instead of T hd^2 on the CUDA cores, whose per-token form passes the whole state through the
// registers' adders twice and needs two block-wide barriers per token. 400 sequences of 322 tokens, one head of 512: 17.5 ms token by
// token, 2.4 ms here (bound by the MMAs and the conversions around them, like efla_seq_kernel).
// ------------------------------------------------------------------------------------------------
constexpr int kLgMaxT = 1024;
constexpr int kLgMat = 4 * kSqTile;                               // the matrix [128][kSqXStride floats]: hi halves, mid halves at kSqPMid
constexpr int kLgDiag = kLgMat + kSeqMaxT * kSqXStride * 4;
constexpr int kLgInv = kLgDiag + 8 * 16 * 17 * 4;
constexpr int kLgScal = kLgInv + 2 * 8 * 16 * kSqTStride * 2;     // q scale, k scale, a, b [4][T]
constexpr int kLgRed = kLgScal + 4 * kLgMaxT * 4;
constexpr int kLgState = kLgRed + 64;
constexpr int kLgSmem = kLgState + 16;
static_assert(2 * kSeqMaxT * kSqLStride * 2 <= 4 * kSqTile, "L takes the staging tiles' place while the diagonal block is inverted");
static_assert(kLgMat % 16 == 0 && kLgDiag % 16 == 0 && kLgInv % 16 == 0 && kLgScal % 16 == 0 && kLgRed % 16 == 0, "16-byte aligned regions");

enum LongOut { LO_WRITE, LO_FROM_V, LO_SUB, LO_ADD };  // out = D, out = b v - D, out -= D, out += D

__global__ void __launch_bounds__(kSeqThreads, 1) efla_long_kernel(const EflaParams p) {
    pdl_wait();
    extern __shared__ __align__(16) uint8_t sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tq = lane & 3;
    const int T = p.T, hd = p.hidden / p.heads;
    const unsigned unit = blockIdx.x;
    const unsigned seq = unit / static_cast<unsigned>(p.heads);
    const int h = static_cast<int>(unit - seq * static_cast<unsigned>(p.heads));
    const int nblocks = (T + kSeqMaxT - 1) / kSeqMaxT, nd = (hd + 63) >> 6;
    const size_t row0 = static_cast<size_t>(seq) * T;
    const float* qg = static_cast<const float*>(p.q) + row0 * p.ld_qkv + h * hd;
    const float* kg = static_cast<const float*>(p.k) + row0 * p.ld_qkv + h * hd;
    const float* vg = static_cast<const float*>(p.v) + row0 * p.ld_qkv + h * hd;
    float* og = static_cast<float*>(p.out) + row0 * p.ld_out + h * hd;
    float* qs_sh = reinterpret_cast<float*>(sm + kLgScal);
    float* ks_sh = qs_sh + kLgMaxT;
    float* a_sh = ks_sh + kLgMaxT;
    float* b_sh = a_sh + kLgMaxT;
    uint32_t* red = reinterpret_cast<uint32_t*>(sm + kLgRed);
    int* state = reinterpret_cast<int*>(sm + kLgState);  // tokens in use; whether a v was no number
    const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(sm));

    // ---------------- norms and scalars of all tokens (as in efla_seq_kernel) ----------------
    for (int t = warp; t < nblocks * kSeqMaxT; t += 16) {
        float qss = 0.0f, kss = 0.0f;
        if (t < T) {
            const float4* q4 = reinterpret_cast<const float4*>(qg + static_cast<size_t>(t) * p.ld_qkv);
            const float4* k4 = reinterpret_cast<const float4*>(kg + static_cast<size_t>(t) * p.ld_qkv);
            for (int i = lane; i < (hd >> 2); i += 32) {
                const float4 a = q4[i], b = k4[i];
                qss = fmaf(a.x, a.x, qss); qss = fmaf(a.y, a.y, qss); qss = fmaf(a.z, a.z, qss); qss = fmaf(a.w, a.w, qss);
                kss = fmaf(b.x, b.x, kss); kss = fmaf(b.y, b.y, kss); kss = fmaf(b.z, b.z, kss); kss = fmaf(b.w, b.w, kss);
            }
        }
        qss = warp_sum_f(qss);
        kss = warp_sum_f(kss);
        if (t < T) kss = seq_infinite_norm(kss, kg + static_cast<size_t>(t) * p.ld_qkv, hd, lane);
        if (lane == 0) { qs_sh[t] = qss; ks_sh[t] = kss; }
    }
    if (tid == 0) { state[0] = T; state[1] = 0; }
    __syncthreads();
    const float bias = efla_seq_bias(p, seq);
    for (int t = tid; t < nblocks * kSeqMaxT; t += kSeqThreads) {
        float a = 0.0f, b = 0.0f, ks = 0.0f, qs = 0.0f;
        if (t < T) seq_scalars(p, p.beta_raw[(row0 + t) * p.ld_beta] + bias, qs_sh[t], ks_sh[t], qs, ks, a, b);
        qs_sh[t] = kSqUp * qs;
        ks_sh[t] = kSqUp * ks;
        a_sh[t] = a;
        b_sh[t] = b;
        if (!(a == a && b == b)) atomicMin(state, t);
    }
    __syncthreads();
    const int Te = state[0];  // tokens before the first one that makes the state NaN
    if (Te < T) {
        for (int t = Te + tid; t < T; t += kSeqThreads) qs_sh[t] = ks_sh[t] = a_sh[t] = b_sh[t] = 0.0f;
        __syncthreads();
    }

    const int piece = tid & 15, srow = tid >> 4;  // staging: 16-byte piece of a 64-column row, rows srow + 32 i
    const int wr = warp >> 1, wc = warp & 1;      // results: 16-row block, column half
    auto load = [&](float4 (&r)[4], const float* base, int ld, int blk, int ct) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = blk * kSeqMaxT + srow + 32 * i, c = ct * 64 + 4 * piece;
            r[i] = t < Te && c < hd ? *reinterpret_cast<const float4*>(base + static_cast<size_t>(t) * ld + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    auto store = [&](const float4 (&r)[4], int tile, const float* scale, float common) {  // two halves per value
        uint8_t* st = sm + tile * kSqTile;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f = scale != nullptr ? scale[srow + 32 * i] : common;
            const int o = ((srow + 32 * i) * kSqStride + 4 * piece) * 2;
            uint2 hi, mid;
            sq_split(r[i].x * f, r[i].y * f, hi.x, mid.x);
            sq_split(r[i].z * f, r[i].w * f, hi.y, mid.y);
            *reinterpret_cast<uint2*>(st + o) = hi;
            *reinterpret_cast<uint2*>(st + kSqTile + o) = mid;
        }
    };

    // rows of block I of `rows` (normalised by rscale) times rows of block J of k; G (is_g: scaled by a, strictly lower on the diagonal) or
    // X (lower on the diagonal). Into the matrix, or (G on the diagonal) L and its diagonal blocks for the inversion.
    auto gram = [&](const float* rows, const float* rscale, bool is_g, int I, int J) {
        float acc[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] = 0.0f;
        float4 ra[4], rb[4];
        load(ra, rows, p.ld_qkv, I, 0);
        load(rb, kg, p.ld_qkv, J, 0);
        const bool used = I != J || wc == 0 || wr >= 4;  // the upper half of a diagonal block is not needed
        const uint32_t aa = sm0 + static_cast<uint32_t>((wr * 16 + (lane & 15)) * kSqStride + (lane >> 4) * 8) * 2u;
        const uint32_t ba = sm0 + 2u * kSqTile + static_cast<uint32_t>((wc * 64 + (lane & 7)) * kSqStride + ((lane >> 3) & 1) * 8) * 2u + (lane >> 4) * static_cast<uint32_t>(kSqTile);
        for (int db = 0; db < nd; ++db) {
            store(ra, 0, rscale + I * kSeqMaxT, 0.0f);
            store(rb, 2, ks_sh + J * kSeqMaxT, 0.0f);
            __syncthreads();
            if (db + 1 < nd) {
                load(ra, rows, p.ld_qkv, I, db + 1);
                load(rb, kg, p.ld_qkv, J, db + 1);
            }
            if (used) {
                const int nk = min(4, (hd - db * 64) >> 4);
                for (int kk = 0; kk < nk; ++kk) {
                    uint32_t ah[4], am[4];
                    ldmatrix_x4(ah, aa + kk * 32);
                    ldmatrix_x4(am, aa + kSqTile + kk * 32);
#pragma unroll
                    for (int n = 0; n < 8; n += 2) {
                        uint32_t b[4], c[4];
                        ldmatrix_x4(b, ba + kk * 32 + n * (8 * kSqStride * 2));
                        ldmatrix_x4(c, ba + kk * 32 + (n + 1) * (8 * kSqStride * 2));
                        mma_f16_16816(acc[n], ah, b[0], b[1]); mma_f16_16816(acc[n + 1], ah, c[0], c[1]);
                        mma_f16_16816(acc[n], ah, b[2], b[3]); mma_f16_16816(acc[n + 1], ah, c[2], c[3]);
                        mma_f16_16816(acc[n], am, b[0], b[1]); mma_f16_16816(acc[n + 1], am, c[0], c[1]);
                    }
                }
            }
            __syncthreads();
        }
        const float gdown = 1.0f / (kSqUp * kSqUp);
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int c0 = wc * 64 + n * 8 + 2 * tq;
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                const int t = wr * 16 + g + 8 * hr;
                const float f = is_g ? gdown * a_sh[I * kSeqMaxT + t] : gdown;
                const int last = I != J ? kSeqMaxT : is_g ? t - 1 : t;  // last column kept
                const float x0 = c0 <= last ? acc[n][2 * hr] * f : 0.0f, x1 = c0 + 1 <= last ? acc[n][2 * hr + 1] * f : 0.0f;
                uint32_t hi, mid;
                sq_split(x0 * kSqUp, x1 * kSqUp, hi, mid);
                if (is_g && I == J) {
                    *reinterpret_cast<uint32_t*>(sm + (t * kSqLStride + c0) * 2) = hi;
                    *reinterpret_cast<uint32_t*>(sm + (kSeqMaxT * kSqLStride + t * kSqLStride + c0) * 2) = mid;
                    if ((c0 >> 4) == wr) {
                        float* d = reinterpret_cast<float*>(sm + kLgDiag) + t * 17 + (c0 & 15);
                        d[0] = x0;
                        d[1] = x1;
                    }
                } else {
                    uint8_t* d = sm + kLgMat + t * (kSqXStride * 4) + c0 * 2;
                    *reinterpret_cast<uint32_t*>(d) = hi;
                    *reinterpret_cast<uint32_t*>(d + kSqPMid) = mid;
                }
            }
        }
        __syncthreads();
    };

    // out block I (op) matrix times block J of src (rows scaled by b where src is v); lower: only the lower triangle of blocks is read
    auto product = [&](const float* src, int ld, bool scale_b, int I, int J, bool lower, LongOut op) {
        float4 r[4];
        auto fetch = [&](int ct) {
            load(r, src, ld, J, ct);
            if (scale_b) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float f = b_sh[J * kSeqMaxT + srow + 32 * i];
                    r[i].x *= f; r[i].y *= f; r[i].z *= f; r[i].w *= f;
                }
            }
        };
        fetch(0);
        const uint32_t pa = sm0 + kLgMat + static_cast<uint32_t>((wr * 16 + (lane & 15)) * (kSqXStride * 4) + (lane >> 4) * 16);
        const uint32_t vb = sm0 + static_cast<uint32_t>(((lane >> 3 & 1) * 8 + (lane & 7)) * kSqStride + wc * 32 + (lane >> 4) * 8) * 2u;
        for (int ct = 0; ct < nd; ++ct) {
            uint32_t m = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) m = max(m, seq_abs_bits(r[i]));
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) red[warp] = m;
            __syncthreads();  // also: everyone is done with the previous tile
            m = __reduce_max_sync(0xffffffffu, red[lane & 15]);
            if (scale_b && m >= kSeqNonFinite) {  // (v: w is finite)
                __syncthreads();  // everyone has read red
                m = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    for (float* x : {&r[i].x, &r[i].y, &r[i].z, &r[i].w})
                        if (!(fabsf(*x) <= FLT_MAX)) *x = 0.0f;
                    m = max(m, seq_abs_bits(r[i]));
                }
                m = __reduce_max_sync(0xffffffffu, m);
                if (lane == 0) red[warp] = m;
                state[1] = 1;
                __syncthreads();
                m = __reduce_max_sync(0xffffffffu, red[lane & 15]);
            }
            const float vs = sq_pow2_scale<15>(__uint_as_float(m));
            store(r, 0, nullptr, vs);
            if (ct + 1 < nd) fetch(ct + 1);
            __syncthreads();
            float y[4][4];
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) y[n][e] = 0.0f;
            const int last = lower ? wr : 7;
            for (int j = 0; j <= last; ++j) {
                uint32_t ah[4], am[4];
                ldmatrix_x4(ah, pa + j * 32);
                ldmatrix_x4(am, pa + kSqPMid + j * 32);
#pragma unroll
                for (int np = 0; np < 2; ++np) {
                    uint32_t vh[4], vm[4];
                    ldmatrix_x4_trans(vh, vb + j * (16 * kSqStride * 2) + np * 32);
                    ldmatrix_x4_trans(vm, vb + kSqTile + j * (16 * kSqStride * 2) + np * 32);
#pragma unroll
                    for (int n = 0; n < 2; ++n) mma_f16_16816(y[2 * np + n], ah, vh[2 * n], vh[2 * n + 1]);
#pragma unroll
                    for (int n = 0; n < 2; ++n) mma_f16_16816(y[2 * np + n], ah, vm[2 * n], vm[2 * n + 1]);
#pragma unroll
                    for (int n = 0; n < 2; ++n) mma_f16_16816(y[2 * np + n], am, vh[2 * n], vh[2 * n + 1]);
                }
            }
            const float ds = 1.0f / kSqUp / vs;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int c = ct * 64 + wc * 32 + n * 8 + 2 * tq;
#pragma unroll
                for (int hr = 0; hr < 2; ++hr) {
                    const int t = I * kSeqMaxT + wr * 16 + g + 8 * hr;
                    if (t >= T || c >= hd) continue;
                    float2* o = reinterpret_cast<float2*>(og + static_cast<size_t>(t) * p.ld_out + c);
                    float2 x = make_float2(y[n][2 * hr] * ds, y[n][2 * hr + 1] * ds);
                    if (op == LO_FROM_V) {
                        float2 v = *reinterpret_cast<const float2*>(vg + static_cast<size_t>(t) * p.ld_qkv + c);
                        if (!(fmaxf(fabsf(v.x), fabsf(v.y)) <= FLT_MAX) || v.x != v.x || v.y != v.y) {
                            if (!(fabsf(v.x) <= FLT_MAX)) v.x = 0.0f;
                            if (!(fabsf(v.y) <= FLT_MAX)) v.y = 0.0f;
                            state[1] = 1;
                        }
                        if (t >= Te) v = make_float2(0.0f, 0.0f);
                        x = make_float2(fmaf(b_sh[t], v.x, -x.x), fmaf(b_sh[t], v.y, -x.y));
                    } else if (op == LO_SUB || op == LO_ADD) {
                        const float2 old = *o;
                        x = op == LO_SUB ? make_float2(old.x - x.x, old.y - x.y) : make_float2(old.x + x.x, old.y + x.y);
                    }
                    *o = x;
                }
            }
        }
        __syncthreads();  // the block is complete, matrix and tile are free
    };

    // inverse of the unit lower triangular I + L of a diagonal block, from its 16 x 16 diagonal blocks outwards, into the matrix
    auto invert = [&] {
        seq_invert_diagonal(reinterpret_cast<const float*>(sm + kLgDiag), reinterpret_cast<__half*>(sm + kLgInv), 8, warp, lane);
        __syncthreads();
        if (warp < 8) {
            seq_solve_rows<32, kSqPMid>(sm0, kLgMat, sm + kLgMat, kLgInv, warp, lane,
                                        [&](int j, int n, int e) { return j == warp && n * 8 + 2 * tq + (e & 1) == g + 8 * (e >> 1) ? 1.0f : 0.0f; });
        }
        __syncthreads();
    };

    for (int I = 0; I < nblocks; ++I) {
        for (int J = 0; J < I; ++J) {
            gram(kg, ks_sh, true, I, J);
            product(og, p.ld_out, false, I, J, false, J == 0 ? LO_FROM_V : LO_SUB);
        }
        gram(kg, ks_sh, true, I, I);
        invert();
        if (I == 0) product(vg, p.ld_qkv, true, 0, 0, true, LO_WRITE);
        else product(og, p.ld_out, false, I, I, true, LO_WRITE);
    }
    for (int I = nblocks - 1; I >= 0; --I) {
        gram(qg, qs_sh, false, I, I);
        product(og, p.ld_out, false, I, I, true, LO_WRITE);
        for (int J = 0; J < I; ++J) {
            gram(qg, qs_sh, false, I, J);
            product(og, p.ld_out, false, I, J, false, LO_ADD);
        }
    }
    if (Te < T || state[1] != 0) {  // (product ends with a barrier)
        for (int c = tid; c < hd; c += kSeqThreads) {
            int t = 0;
            while (t < Te && fabsf(vg[static_cast<size_t>(t) * p.ld_qkv + c]) <= FLT_MAX) ++t;
            for (; t < T; ++t) og[static_cast<size_t>(t) * p.ld_out + c] = NAN;
        }
    }
}

}  // namespace

// Do the addresses from the output's first to its last lie apart from those of q, k or v?
static bool seq_ranges_apart(const EflaParams& p, const void* in) {
    if (p.seqs <= 0) return true;
    const size_t last = static_cast<size_t>(p.seqs) * p.T - 1;
    const char *o = static_cast<const char*>(p.out), *a = static_cast<const char*>(in);
    return o >= a + (last * p.ld_qkv + p.hidden) * sizeof(float) || a >= o + (last * p.ld_out + p.hidden) * sizeof(float);
}
static SeqOverlap seq_overlap(const EflaParams& p, const void* in) {
    if (seq_ranges_apart(p, in)) return SEQ_APART;
    if (p.ld_out != p.ld_qkv) return SEQ_ACROSS;
    if (in == p.out) return SEQ_SAME;
    const long long row = static_cast<long long>(p.ld_qkv) * sizeof(float), width = static_cast<long long>(p.hidden) * sizeof(float);
    if (row < 2 * width) return SEQ_ACROSS;
    const long long d = ((static_cast<long long>(reinterpret_cast<intptr_t>(p.out)) - static_cast<long long>(reinterpret_cast<intptr_t>(in))) % row + row) % row;
    return d < width ? SEQ_RIGHT : row - d < width ? SEQ_ACROSS : SEQ_APART;
}

// The closed form's work per token grows with the sequence, the per-token kernel's does not, but the latter spreads a unit over several SMs. One head of
// 512: 322 tokens 0.69 / 1.16 ms (closed form / per token) for 4 sequences, 2.4 / 17.5 ms for 400; 1000 tokens 4.4 / 3.6 ms for 4, 5.0 / 8.3 ms for 40.
// The number of sequences has no say: the two round differently, and a member's loss must not depend on how many share its wave.
static bool seq_long_pays(const EflaParams& p) {
    return p.T <= kLgMaxT && seq_ranges_apart(p, p.q) && seq_ranges_apart(p, p.k) && seq_ranges_apart(p, p.v);  // (the output holds w before all of them have been read)
}

// (heads of 32 are faster one warp each, token by token: efla_head32_kernel)
bool efla_seq_applies(const EflaParams& p) {
    const int hd = p.hidden / p.heads;
    return p.state == nullptr && p.state_fp16 != 0 && !p.qkv_f16 && !p.out_f16 && hd > 32 && hd % 32 == 0 && (p.T <= kSeqMaxT || (seq_long_pays(p) && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0 && p.ld_out % 4 == 0)) &&
           ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v)) & 15) == 0 && p.ld_qkv % 4 == 0 &&
           (reinterpret_cast<uintptr_t>(p.out) & 7) == 0 && p.ld_out % 2 == 0 && p.seqs * static_cast<long long>(p.heads) <= 0x7fffffffLL / 4;
}

int efla_seq_launch(const EflaParams& p, cudaStream_t stream) {
    int dev = 0;
    const int rc = current_device(&dev);
    if (rc) return rc;
    const long long units = p.seqs * p.heads;
    if (p.T > kSeqMaxT) {
        static std::atomic<bool> configured[64] = {};  // function attributes are per device
        if (dev >= 64 || !configured[dev].load(std::memory_order_relaxed)) {
            const int rc2 = check_cuda(cudaFuncSetAttribute(efla_long_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLgSmem), "cudaFuncSetAttribute(efla_long_kernel)");
            if (rc2) return rc2;
            if (dev < 64) configured[dev].store(true, std::memory_order_relaxed);
        }
        launch_pdl_if(false, efla_long_kernel, static_cast<unsigned>(units), kSeqThreads, kLgSmem, stream, p);
        return check_launch("efla_long_kernel");
    }
    static std::atomic<bool> configured[64] = {};
    if (dev >= 64 || !configured[dev].load(std::memory_order_relaxed)) {
        const int rc2 = check_cuda(cudaFuncSetAttribute(efla_seq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSqSmem), "cudaFuncSetAttribute(efla_seq_kernel)");
        if (rc2) return rc2;
        if (dev < 64) configured[dev].store(true, std::memory_order_relaxed);
    }
    // Few units leave SMs idle: two or four CTAs each take a share of a unit's column tiles, as long as all run at once (the sums before them are done by
    // each). One head of 512, 128 tokens: 32 sequences 34.7 us with one CTA each, 27.2 with four; 70 sequences 35.3 with one, 30.3 with two; 32 of 16 tokens 24.4 and 18.2. Where the output lies on q or k, the CTAs of
    // a unit are a cluster; fours of them fit all SMs of a chip only in part (a processing cluster of 18 SMs holds four).
    const int sms = multiprocessors(dev), nd = (p.hidden / p.heads + 63) >> 6;
    if (sms <= 0) return BNF4_ERR_CUDA;
    const bool meet = seq_overlap(p, p.q) != SEQ_APART || seq_overlap(p, p.k) != SEQ_APART;
    const SeqOverlap across = seq_overlap(p, p.v);
    const int cs = across == SEQ_RIGHT || across == SEQ_ACROSS ? 1 : units * 4 <= (meet ? sms * 7 / 8 : sms) && nd >= 4 ? 4 : units * 2 <= sms && nd >= 2 ? 2 : 1;
    const bool early = p.seqs * static_cast<long long>(p.T) * p.hidden <= kPdlStreamElems;
    CUtensorMap maps[3];  // boxes of a sequence's tokens and 32 columns (boxes of 128 tokens always: 500 sequences of 33 on three heads of 96 136 us, 130 so)
    const void* in[3] = {p.q, p.k, p.v};
    for (int i = 0; i < 3; ++i) {
        const int rc2 = make_map_2d(&maps[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, in[i], static_cast<uint64_t>(p.hidden), static_cast<uint64_t>(p.seqs) * static_cast<uint64_t>(p.T),
                                    static_cast<uint64_t>(p.ld_qkv) * 4, 32, static_cast<uint32_t>(p.T), "scan inputs");
        if (rc2) return rc2;
    }
    if (cs > 1 && meet) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(units * cs));
        cfg.blockDim = dim3(kSqThreads);
        cfg.dynamicSmemBytes = kSqSmem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(cs);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = early ? 2 : 1;
        cudaLaunchKernelEx(&cfg, efla_seq_kernel, maps[0], maps[1], maps[2], p, cs, 1, static_cast<int>(across));  // errors surface in check_launch
    } else {
        launch_pdl_if(early, efla_seq_kernel, static_cast<unsigned>(units * cs), kSqThreads, kSqSmem, stream, maps[0], maps[1], maps[2], p, cs, 0, static_cast<int>(across));
    }
    return check_launch("efla_seq_kernel");
}

int efla_seq_device_error(int* code) { return take_wait_error(code); }

}  // namespace bnf4
