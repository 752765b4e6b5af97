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
// Precision: every operand is split into two fp16 terms (x = hi + mid, 22 significant bits; rows are normalised and scaled by powers of
// two first so that neither term under- or overflows) and the products hi hi + hi mid + mid hi accumulate in fp32. Nothing is
// rounded to fp16 between tokens, so the result lies closer to exact arithmetic than the per-token form's fp16 state.
//
// Values that are no numbers stay where the recurrence has them, although 0 x NaN is NaN in a contraction: from the first token on whose k or beta
// makes the state NaN, the sequence is cut off (as if it ended there) and the rows behind it are NaN; a v that is no number is taken out
// and its column is NaN from its token on; in q it only meets its own row.
//
// One CTA of 16 warps per (sequence, head):
//   1. norms of q and k and the per-token scalars (one warp per row),
//   2. G and X = Q^ K^^T over 64-column blocks of K and Q (fp32 -> two halves -> shared memory, double-buffered, the next block's
//      loads in flight behind the MMAs). Warp (pair, G or X, column half) owns row blocks p and nb - 1 - p, so the lower
//      triangles are spread evenly,
//   3. inverses of the 16 x 16 diagonal blocks of I + diag(a) strict(G) by forward substitution in fp32,
//   4. P~ by block back substitution from the right, one warp per 16-row block (rows are independent, no barriers),
//   5. y = P~ V over 64-column tiles of V.
// What bounds it: the MMAs of steps 2 and 5 (about 40 k tensor cycles per sequence at T = 128, hd = 512; the legacy mma.sync path, since
// the triangular solve between the contractions needs its operands in registers). 1024 sequences of 128 tokens, one head of 512:
// 0.56 ms, against 17.6 ms for the per-token kernel. Of 150 k cycles per unit, step 1
// takes 31 k (DRAM), step 2 63 k, steps 3 and 4 8 k, step 5 47 k. MMAs and the conversions around them add up rather than overlap: staggering them
// between warps, more independent MMA chains and L2 prefetches of V and of the next unit changed nothing.

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace bnf4 {

namespace {

constexpr int kSeqMaxT = 128;
constexpr int kSeqThreads = 512;
constexpr int kSqStride = 72;                      // halves per row of the K / Q / V blocks: conflict-free ldmatrix rows
constexpr int kSqTile = kSeqMaxT * kSqStride * 2;  // bytes of one 128 x 64 block of halves
constexpr int kSqStage = 4 * kSqTile;              // K hi, K mid, Q hi, Q mid
constexpr int kSqLStride = 136;                    // halves per row of L hi / L mid
constexpr int kSqXStride = 140;                    // floats per row of X; the row then holds P~ hi (272 bytes) and P~ mid
constexpr int kSqPMid = 272;                       // byte offset of P~ mid inside a row
constexpr int kSqTStride = 24;                     // halves per row of a diagonal block's inverse
constexpr int kSqDiag = 2 * kSqStage;                            // fp32 diagonal blocks of L [8][16][17]
constexpr int kSqInv = kSqDiag + 8 * 16 * 17 * 4;                // their inverses, hi and mid [2][8][16][kSqTStride]
constexpr int kSqScal = kSqInv + 2 * 8 * 16 * kSqTStride * 2;    // q scale, k scale, a, b [4][128] floats
constexpr int kSqRed = kSqScal + 4 * kSeqMaxT * 4;               // reduction scratch [2][16] + broadcast
constexpr int kSqPart = kSqRed + 256;                            // squared norms of a CTA's tokens [2][128] floats (read by its cluster)
constexpr int kSqBad = kSqPart + 2 * kSeqMaxT * 4;               // first token of each of 64 columns whose v is no number
constexpr int kSqSmem = kSqBad + 64 * 4;
static_assert(2 * kSeqMaxT * kSqLStride * 2 <= kSqStage && kSeqMaxT * kSqXStride * 4 <= kSqStage && 4 * kSqTile <= kSqStage, "overlaid regions");
static_assert(kSqDiag % 16 == 0 && kSqInv % 16 == 0 && kSqScal % 16 == 0, "16-byte aligned regions");
constexpr float kSqUp = 256.0f;                    // power-of-two scale of every normalised operand

__device__ __forceinline__ void sq_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void sq_ldm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void sq_ldm_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
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

// One warp: rows 16 i .. 16 i + 15 of P with P (I + L) = X by block columns from the right; X in registers, L (two halves) at the start of
// shared memory, the diagonal blocks' inverses at inv_off; P (two halves, scaled by kSqUp) at mat_off (prow: the same place).
__device__ __forceinline__ void seq_solve_rows(uint32_t sm0, uint32_t mat_off, uint8_t* prow, uint32_t inv_off, int i, int lane, const float (&xr)[8][2][4]) {
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
            sq_ldm(ph, p_addr + k * 32);
            sq_ldm(pm, p_addr + kSqPMid + k * 32);
            sq_ldm_trans(lh, l_addr + k * (16 * kSqLStride * 2) + j * 32);
            sq_ldm_trans(lm, l_addr + kLMid + k * (16 * kSqLStride * 2) + j * 32);
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                sq_mma(s[n], ph, lh[2 * n], lh[2 * n + 1]);
                sq_mma(c[n], ph, lm[2 * n], lm[2 * n + 1]);
                sq_mma(c[n], pm, lh[2 * n], lh[2 * n + 1]);
            }
        }
        // z = X_ij - sum, then P~_ij = z inv_jj
        uint32_t zh[4], zm[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            float z[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) z[e] = (xr[j][n][e] - (s[n][e] + c[n][e]) * down) * kSqUp;
            sq_split(z[0], z[1], zh[2 * n], zm[2 * n]);
            sq_split(z[2], z[3], zh[2 * n + 1], zm[2 * n + 1]);
        }
        uint32_t th[4], tm[4];
        sq_ldm_trans(th, i_addr + j * (16 * kSqTStride * 2));
        sq_ldm_trans(tm, i_addr + kIMid + j * (16 * kSqTStride * 2));
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            float o[4] = {0.0f, 0.0f, 0.0f, 0.0f}, oc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            sq_mma(o, zh, th[2 * n], th[2 * n + 1]);
            sq_mma(oc, zh, tm[2 * n], tm[2 * n + 1]);
            sq_mma(oc, zm, th[2 * n], th[2 * n + 1]);
            const int c0 = j * 16 + n * 8 + 2 * tq;
#pragma unroll
            for (int hr = 0; hr < 2; ++hr) {
                uint32_t hi, mid;
                sq_split((o[2 * hr] + oc[2 * hr]) * (1.0f / kSqUp), (o[2 * hr + 1] + oc[2 * hr + 1]) * (1.0f / kSqUp), hi, mid);
                uint8_t* d = prow + (i * 16 + g + 8 * hr) * (kSqXStride * 4) + c0 * 2;
                *reinterpret_cast<uint32_t*>(d) = hi;
                *reinterpret_cast<uint32_t*>(d + kSqPMid) = mid;
            }
        }
        __syncwarp();
    }
}

template <int CS>
__device__ __forceinline__ void sq_cluster_sync() {
    if constexpr (CS > 1) __syncwarp();
    if constexpr (CS > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the float at this shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ float sq_remote(uint32_t addr, int rank) {
    uint32_t a;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// the 16 bytes at this shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ uint4 sq_remote16(uint32_t addr, int rank) {
    uint32_t a;
    uint4 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}

// CS CTAs of a cluster share a unit. No sum is split: a CTA takes some of the tokens in step 1, some of the 16-row blocks of G and X in step 2 (all of
// K, its own rows of Q; finished rows are exchanged through distributed shared memory) and some of the 64-column blocks in step 5; steps 3
// and 4 are done by every one. Every CS gives the same bits, so a sequence's outputs do not depend on how many share the launch.
template <int CS>
__global__ void __launch_bounds__(kSeqThreads, 1) efla_seq_kernel(const EflaParams p) {
    pdl_wait();
    extern __shared__ __align__(16) uint8_t sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int T = p.T, hd = p.hidden / p.heads;
    const unsigned unit = blockIdx.x / CS;
    const int rank = static_cast<int>(blockIdx.x % CS);
    const int nd = (p.hidden / p.heads + 63) >> 6;
    const int db0 = rank * nd / CS, db1 = (rank + 1) * nd / CS;  // this CTA's 64-column blocks
    const unsigned seq = unit / static_cast<unsigned>(p.heads);
    const int h = static_cast<int>(unit - seq * static_cast<unsigned>(p.heads));
    const int nb = (T + 15) >> 4;  // 16-token blocks
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
    int* bad_col = reinterpret_cast<int*>(sm + kSqBad);
    float* part = reinterpret_cast<float*>(sm + kSqPart);
    const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(sm));

    // ---------------- 1. norms and scalars ----------------
    for (int t = warp * CS + rank; t < kSeqMaxT; t += 16 * CS) {
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
        if (lane == 0) { part[t] = qss; part[kSeqMaxT + t] = kss; }
    }
    if constexpr (CS > 1) sq_cluster_sync<CS>();
    else __syncthreads();
    if (tid < kSeqMaxT) {
        const int t = tid;
        float qss = 0.0f, kss = 0.0f;
        if constexpr (CS > 1) {
            qss = sq_remote(sm0 + kSqPart + t * 4, t % CS);
            kss = sq_remote(sm0 + kSqPart + (kSeqMaxT + t) * 4, t % CS);
        } else {
            qss = part[t];
            kss = part[kSeqMaxT + t];
        }
        float a = 0.0f, b = 0.0f, kinv = 0.0f, qinv = 0.0f;
        if (t < T) {
            const float bias = efla_seq_bias(p, static_cast<unsigned>(seq));
            seq_scalars(p, p.beta_raw[(row0 + t) * p.ld_beta] + bias, qss, kss, qinv, kinv, a, b);
        }
        qs_sh[t] = kSqUp * qinv;
        ks_sh[t] = kSqUp * kinv;
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
        if (tid >= Te && tid < T) qs_sh[tid] = ks_sh[tid] = a_sh[tid] = b_sh[tid] = 0.0f;
        __syncthreads();
    }
    const float bscale = sq_pow2_scale<6>(fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3])));  // b * bscale < 64: P~ below 2^14, also for V's sake

    // ---------------- 2. G and X ----------------
    const int pr = rank + CS * ((warp & 3) % (4 / CS)), which = (warp >> 2) & 1, half = warp >> 3;
    const int jq = (warp & 3) / (4 / CS);  // column blocks jq, jq + CS, ..
    const int r1 = pr, r2 = nb - 1 - pr;   // this warp's row blocks (r1 < r2: both; equal: one; r1 > r2: none)
    auto owner = [&](int block) { return min(block, nb - 1 - block) % CS; };  // the CTA that forms this row block
    float acc1[4 / CS][4], acc2[8 / CS][4];
#pragma unroll
    for (int j = 0; j < 8 / CS; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) { acc2[j][i] = 0.0f; if (j < 4 / CS) acc1[j % (4 / CS)][i] = 0.0f; }

    // staging: thread = (16-byte piece of a 64-column row block, row); four rows of K and of Q per thread
    const int piece = tid & 15, srow = tid >> 4;
    float4 kr[4], qr[4];
    auto load_block = [&](int d0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = srow + 32 * i, c = d0 + 4 * piece;
            kr[i] = qr[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (t < Te && c < hd) {
                kr[i] = *reinterpret_cast<const float4*>(kg + static_cast<size_t>(t) * p.ld_qkv + c);
                if (CS == 1 || owner(t >> 4) == rank) qr[i] = *reinterpret_cast<const float4*>(qg + static_cast<size_t>(t) * p.ld_qkv + c);
            }
        }
    };
    auto store_block = [&](int buf) {
        uint8_t* st = sm + buf * kSqStage;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = srow + 32 * i;
            const float ks = ks_sh[t], qs = qs_sh[t];
            const int o = (t * kSqStride + 4 * piece) * 2;
            uint2 hi, mid;
            sq_split(kr[i].x * ks, kr[i].y * ks, hi.x, mid.x);
            sq_split(kr[i].z * ks, kr[i].w * ks, hi.y, mid.y);
            *reinterpret_cast<uint2*>(st + o) = hi;
            *reinterpret_cast<uint2*>(st + kSqTile + o) = mid;
            if (CS > 1 && owner(t >> 4) != rank) continue;
            sq_split(qr[i].x * qs, qr[i].y * qs, hi.x, mid.x);
            sq_split(qr[i].z * qs, qr[i].w * qs, hi.y, mid.y);
            *reinterpret_cast<uint2*>(st + 2 * kSqTile + o) = hi;
            *reinterpret_cast<uint2*>(st + 3 * kSqTile + o) = mid;
        }
    };
    // ldmatrix addresses inside a stage: A rows (lane % 16, column half lane / 16); B: eight K rows, matrices (hi, k 0-7), (hi, 8-15), (mid, ..), (mid, ..)
    const uint32_t a_off = static_cast<uint32_t>((lane & 15) * kSqStride + (lane >> 4) * 8) * 2u + (which ? 2u * kSqTile : 0u);
    const uint32_t b_off = static_cast<uint32_t>((half * 8 + (lane & 7)) * kSqStride + ((lane >> 3) & 1) * 8) * 2u + (lane >> 4) * static_cast<uint32_t>(kSqTile);
    load_block(0);
    store_block(0);
    __syncthreads();
    for (int db = 0; db < nd; ++db) {
        if (db + 1 < nd) load_block((db + 1) * 64);
        const uint32_t st = sm0 + (db & 1) * kSqStage;
        const int nk = min(4, (hd - db * 64) >> 4);
        if (r1 <= r2) {
            for (int kk = 0; kk < nk; ++kk) {
                uint32_t ah1[4], am1[4], ah2[4], am2[4];
                const uint32_t ab = st + a_off + kk * 32;
                sq_ldm(ah2, ab + r2 * (16 * kSqStride * 2));
                sq_ldm(am2, ab + r2 * (16 * kSqStride * 2) + kSqTile);
                sq_ldm(ah1, ab + r1 * (16 * kSqStride * 2));
                sq_ldm(am1, ab + r1 * (16 * kSqStride * 2) + kSqTile);
#pragma unroll
                for (int jj = 0; jj < 8 / CS; ++jj) {
                    const int j = jq + CS * jj;
                    constexpr int N1 = 4 / CS;
                    if (j <= r2) {
                        uint32_t b[4];
                        sq_ldm(b, st + b_off + kk * 32 + j * (16 * kSqStride * 2));
                        sq_mma(acc2[jj], ah2, b[0], b[1]);
                        if (jj < N1 && j <= r1) sq_mma(acc1[jj % N1], ah1, b[0], b[1]);
                        sq_mma(acc2[jj], ah2, b[2], b[3]);
                        if (jj < N1 && j <= r1) sq_mma(acc1[jj % N1], ah1, b[2], b[3]);
                        sq_mma(acc2[jj], am2, b[0], b[1]);
                        if (jj < N1 && j <= r1) sq_mma(acc1[jj % N1], am1, b[0], b[1]);
                    }
                }
            }
        }
        if (db + 1 < nd) store_block((db + 1) & 1);
        __syncthreads();
    }

    // ---------------- 3. L (two halves, stage 0), its diagonal blocks (fp32), X (fp32, stage 1) ----------------
    const int g = lane >> 2, tq = lane & 3;
    __half* Lh = reinterpret_cast<__half*>(sm);
    __half* Lm = Lh + kSeqMaxT * kSqLStride;
    float* X = reinterpret_cast<float*>(sm + kSqStage);
    float* Ld = reinterpret_cast<float*>(sm + kSqDiag);
    const float gdown = 1.0f / (kSqUp * kSqUp);
    auto put_tile = [&](const float (&acc)[4], int r, int j) {
        const int c0 = j * 16 + half * 8 + 2 * tq;
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            const int t = r * 16 + g + 8 * hr;
            float x0 = acc[2 * hr] * gdown, x1 = acc[2 * hr + 1] * gdown;
            if (which == 0) {
                const float at = a_sh[t];
                x0 = c0 < t ? at * x0 : 0.0f;
                x1 = c0 + 1 < t ? at * x1 : 0.0f;
                uint32_t hi, mid;
                sq_split(x0 * kSqUp, x1 * kSqUp, hi, mid);
                *reinterpret_cast<uint32_t*>(Lh + t * kSqLStride + c0) = hi;
                *reinterpret_cast<uint32_t*>(Lm + t * kSqLStride + c0) = mid;
                if (r == j) {
                    float* d = Ld + (r * 16 + g + 8 * hr) * 17 + half * 8 + 2 * tq;
                    d[0] = x0;
                    d[1] = x1;
                }
            } else {
                *reinterpret_cast<float2*>(X + t * kSqXStride + c0) = make_float2(c0 <= t ? x0 : 0.0f, c0 + 1 <= t ? x1 : 0.0f);
            }
        }
    };
#pragma unroll
    for (int jj = 0; jj < 8 / CS; ++jj) {
        const int j = jq + CS * jj;
        if (r1 <= r2 && j <= r2) put_tile(acc2[jj], r2, j);
        if (jj < 4 / CS && r1 < r2 && j <= r1) put_tile(acc1[jj % (4 / CS)], r1, j);
    }
    if constexpr (CS > 1) {  // the other CTAs' rows: L hi and mid, X up to the diagonal block, and that block
        sq_cluster_sync<CS>();
        for (int t = warp; t < 16 * nb; t += 16) {
            const int blk = t >> 4, o = owner(blk);
            if (o == rank) continue;
            const int n2 = 2 * (blk + 1);  // 16-byte pieces of a row of halves
            for (int i = lane; i < 4 * n2; i += 32) {
                const uint32_t at = i < n2 ? (t * kSqLStride) * 2 + i * 16 : i < 2 * n2 ? ((kSeqMaxT + t) * kSqLStride) * 2 + (i - n2) * 16
                                                                                         : kSqStage + (t * kSqXStride) * 4 + (i - 2 * n2) * 16;
                *reinterpret_cast<uint4*>(sm + at) = sq_remote16(sm0 + at, o);
            }
        }
        for (int i = tid; i < nb * 68; i += kSeqThreads) {  // 16 x 17 floats a block
            const int o = owner(i / 68);
            if (o != rank) *reinterpret_cast<uint4*>(sm + kSqDiag + i * 16) = sq_remote16(sm0 + kSqDiag + i * 16, o);
        }
        sq_cluster_sync<CS>();  // everyone has read (and nobody's shared memory is read from here on)
    } else __syncthreads();
    // inverse of I + L_ii: lane c owns column c of a block, two blocks per warp
    seq_invert_diagonal(Ld, reinterpret_cast<__half*>(sm + kSqInv), nb, warp, lane);
    __syncthreads();

    // ---------------- 4. P~ M = X by block columns from the right; warp i owns rows 16 i .. 16 i + 15 ----------------
    // ldmatrix addresses: A rows of P~ (stage 1), B = rows of L / inverse read transposed (matrices (k 0-7, n 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15))
    if (warp < nb) {
        const int i = warp;
        float xr[8][2][4];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j <= i) {
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const float2 lo = *reinterpret_cast<const float2*>(X + (i * 16 + g) * kSqXStride + j * 16 + n * 8 + 2 * tq);
                    const float2 hi = *reinterpret_cast<const float2*>(X + (i * 16 + g + 8) * kSqXStride + j * 16 + n * 8 + 2 * tq);
                    xr[j][n][0] = lo.x; xr[j][n][1] = lo.y; xr[j][n][2] = hi.x; xr[j][n][3] = hi.y;
                }
            }
        }
        __syncwarp();  // the rows are in registers: P~ takes their place
        uint8_t* prow = sm + kSqStage;
        seq_solve_rows(sm0, kSqStage, prow, kSqInv, i, lane, xr);
        // the columns' factors b_s, scaled to at most 64: applied to the finished rows (exact powers of two aside, one more rounding)
        for (int idx = lane; idx < 16 * (i + 1) * 8; idx += 32) {
            const int rr = idx / ((i + 1) * 8), cc = (idx - rr * ((i + 1) * 8)) * 2;
            uint8_t* d = prow + (i * 16 + rr) * (kSqXStride * 4) + cc * 2;
            const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(d)), mf = __half22float2(*reinterpret_cast<const __half2*>(d + kSqPMid));
            uint32_t hi, mid;
            sq_split((hf.x + mf.x) * (b_sh[cc] * bscale), (hf.y + mf.y) * (b_sh[cc + 1] * bscale), hi, mid);
            *reinterpret_cast<uint32_t*>(d) = hi;
            *reinterpret_cast<uint32_t*>(d + kSqPMid) = mid;
        }
    }
    __syncthreads();

    // ---------------- 5. y = P~ V, 64 columns at a time ----------------
    const int cg = warp >> 2;                        // 16-column group of the tile
    const int y1r = warp & 3, y2r = nb - 1 - y1r;    // this warp's row blocks, as r1 and r2 of one CTA per unit
    const uint32_t pa = sm0 + kSqStage + static_cast<uint32_t>((lane & 15) * (kSqXStride * 4) + (lane >> 4) * 16);
    const uint32_t vb = sm0 + static_cast<uint32_t>(((lane >> 3 & 1) * 8 + (lane & 7)) * kSqStride + cg * 16 + (lane >> 4) * 8) * 2u;
    float4 vr[4];
    auto load_v = [&](int c0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = srow + 32 * i, c = c0 + 4 * piece;
            vr[i] = (t < Te && c < hd) ? *reinterpret_cast<const float4*>(vg + static_cast<size_t>(t) * p.ld_qkv + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    load_v(db0 * 64);
    for (int ct = db0; ct < db1; ++ct) {
        // the tile's own power-of-two scale keeps both halves of its values in range
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) m = max(m, seq_abs_bits(vr[i]));
        m = __reduce_max_sync(0xffffffffu, m);
        uint32_t* redb = reinterpret_cast<uint32_t*>(red) + 16 * (ct & 1);
        if (lane == 0) redb[warp] = m;
        __syncthreads();  // also: everyone is done with the tile before the previous one
        m = __reduce_max_sync(0xffffffffu, redb[lane & 15]);
        const bool tile_bad = m >= kSeqNonFinite;
        if (tile_bad) {
            if (tid < 64) bad_col[tid] = T;
            __syncthreads();
            m = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                auto clear = [&](float& x, int e) {
                    if (!(fabsf(x) <= FLT_MAX)) {
                        atomicMin(bad_col + 4 * piece + e, srow + 32 * i);
                        x = 0.0f;
                    }
                };
                clear(vr[i].x, 0); clear(vr[i].y, 1); clear(vr[i].z, 2); clear(vr[i].w, 3);
                m = max(m, seq_abs_bits(vr[i]));
            }
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) redb[warp] = m;  // (read by everyone before the barrier above)
            __syncthreads();
            m = __reduce_max_sync(0xffffffffu, redb[lane & 15]);
        }
        const float vs = sq_pow2_scale<15>(__uint_as_float(m));
        uint8_t* st = sm + (ct & 1) * (2 * kSqTile);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int o = ((srow + 32 * i) * kSqStride + 4 * piece) * 2;
            uint2 hi, mid;
            sq_split(vr[i].x * vs, vr[i].y * vs, hi.x, mid.x);
            sq_split(vr[i].z * vs, vr[i].w * vs, hi.y, mid.y);
            *reinterpret_cast<uint2*>(st + o) = hi;
            *reinterpret_cast<uint2*>(st + kSqTile + o) = mid;
        }
        if (ct + 1 < db1) load_v((ct + 1) * 64);
        __syncthreads();
        if (y1r <= y2r) {
            float y1[2][4], y2[2][4];
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) y1[n][e] = y2[n][e] = 0.0f;
            const uint32_t vbt = vb + (ct & 1) * (2 * kSqTile);
            for (int j = 0; j <= y2r; ++j) {
                uint32_t vh[4], vm[4], ah[4], am[4];
                sq_ldm_trans(vh, vbt + j * (16 * kSqStride * 2));
                sq_ldm_trans(vm, vbt + kSqTile + j * (16 * kSqStride * 2));
                sq_ldm(ah, pa + y2r * (16 * kSqXStride * 4) + j * 32);
                sq_ldm(am, pa + y2r * (16 * kSqXStride * 4) + kSqPMid + j * 32);
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    sq_mma(y2[n], ah, vh[2 * n], vh[2 * n + 1]);
                    sq_mma(y2[n], ah, vm[2 * n], vm[2 * n + 1]);
                    sq_mma(y2[n], am, vh[2 * n], vh[2 * n + 1]);
                }
                if (y1r < y2r && j <= y1r) {
                    sq_ldm(ah, pa + y1r * (16 * kSqXStride * 4) + j * 32);
                    sq_ldm(am, pa + y1r * (16 * kSqXStride * 4) + kSqPMid + j * 32);
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        sq_mma(y1[n], ah, vh[2 * n], vh[2 * n + 1]);
                        sq_mma(y1[n], ah, vm[2 * n], vm[2 * n + 1]);
                        sq_mma(y1[n], am, vh[2 * n], vh[2 * n + 1]);
                    }
                }
            }
            // undo the scales of P~ (2^8 and b's) and of V
            const float ds = 1.0f / kSqUp / bscale / vs;
            auto put = [&](const float (&y)[2][4], int r) {
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const int c = ct * 64 + cg * 16 + n * 8 + 2 * tq;
#pragma unroll
                    for (int hr = 0; hr < 2; ++hr) {
                        const int t = r * 16 + g + 8 * hr;
                        float2 x = make_float2(y[n][2 * hr] * ds, y[n][2 * hr + 1] * ds);
                        if (tile_bad || Te < T) {
                            if (t >= Te || (tile_bad && t >= bad_col[c & 63])) x.x = NAN;
                            if (t >= Te || (tile_bad && t >= bad_col[(c & 63) + 1])) x.y = NAN;
                        }
                        if (t < T && c < hd) *reinterpret_cast<float2*>(og + static_cast<size_t>(t) * p.ld_out + c) = x;
                    }
                }
            };
            put(y2, y2r);
            if (y1r < y2r) put(y1, y1r);
        }
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
                    sq_ldm(ah, aa + kk * 32);
                    sq_ldm(am, aa + kSqTile + kk * 32);
#pragma unroll
                    for (int n = 0; n < 8; n += 2) {
                        uint32_t b[4], c[4];
                        sq_ldm(b, ba + kk * 32 + n * (8 * kSqStride * 2));
                        sq_ldm(c, ba + kk * 32 + (n + 1) * (8 * kSqStride * 2));
                        sq_mma(acc[n], ah, b[0], b[1]); sq_mma(acc[n + 1], ah, c[0], c[1]);
                        sq_mma(acc[n], ah, b[2], b[3]); sq_mma(acc[n + 1], ah, c[2], c[3]);
                        sq_mma(acc[n], am, b[0], b[1]); sq_mma(acc[n + 1], am, c[0], c[1]);
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
                sq_ldm(ah, pa + j * 32);
                sq_ldm(am, pa + kSqPMid + j * 32);
#pragma unroll
                for (int np = 0; np < 2; ++np) {
                    uint32_t vh[4], vm[4];
                    sq_ldm_trans(vh, vb + j * (16 * kSqStride * 2) + np * 32);
                    sq_ldm_trans(vm, vb + kSqTile + j * (16 * kSqStride * 2) + np * 32);
#pragma unroll
                    for (int n = 0; n < 2; ++n) sq_mma(y[2 * np + n], ah, vh[2 * n], vh[2 * n + 1]);
#pragma unroll
                    for (int n = 0; n < 2; ++n) sq_mma(y[2 * np + n], ah, vm[2 * n], vm[2 * n + 1]);
#pragma unroll
                    for (int n = 0; n < 2; ++n) sq_mma(y[2 * np + n], am, vh[2 * n], vh[2 * n + 1]);
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
            float xr[8][2][4];
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) xr[j][n][e] = j == warp && n * 8 + 2 * tq + (e & 1) == g + 8 * (e >> 1) ? 1.0f : 0.0f;
            seq_solve_rows(sm0, kLgMat, sm + kLgMat, kLgInv, warp, lane, xr);
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

// The closed form's work per token grows with the sequence, the per-token kernel's does not, but the latter spreads a unit over several SMs. One head of
// 512: 322 tokens 0.69 / 1.16 ms (closed form / per token) for 4 sequences, 2.4 / 17.5 ms for 400; 1000 tokens 4.4 / 3.6 ms for 4, 5.0 / 8.3 ms for 40.
// The number of sequences has no say: the two round differently, and a member's loss must not depend on how many share its wave.
static bool seq_long_pays(const EflaParams& p) {
    if (p.T > kLgMaxT) return false;
    // the output holds w before all of q, k and v have been read: it must not lie among them
    if (p.seqs <= 0) return true;
    const size_t last = static_cast<size_t>(p.seqs) * p.T - 1;
    const char* o = static_cast<const char*>(p.out);
    const char* o_end = o + (last * p.ld_out + p.hidden) * sizeof(float);
    for (const void* in : {static_cast<const void*>(p.q), static_cast<const void*>(p.k), static_cast<const void*>(p.v)}) {
        const char* a = static_cast<const char*>(in);
        if (o < a + (last * p.ld_qkv + p.hidden) * sizeof(float) && a < o_end) return false;
    }
    return true;
}

// (heads of 32 are faster one warp each, token by token: efla_head32_kernel)
bool efla_seq_applies(const EflaParams& p) {
    const int hd = p.hidden / p.heads;
    return p.state == nullptr && p.state_fp16 != 0 && !p.qkv_f16 && !p.out_f16 && hd > 32 && hd % 32 == 0 && (p.T <= kSeqMaxT || (seq_long_pays(p) && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0 && p.ld_out % 4 == 0)) &&
           ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v)) & 15) == 0 && p.ld_qkv % 4 == 0 &&
           (reinterpret_cast<uintptr_t>(p.out) & 7) == 0 && p.ld_out % 2 == 0 && p.seqs * static_cast<long long>(p.heads) <= 0x7fffffffLL / 4;
}

namespace {
// Clusters of CS such CTAs that the device holds at once (a cluster stays inside one processing cluster of the chip: fewer than SMs / CS); 0 on error.
template <int CS>
int resident_clusters(int dev) {
    static std::atomic<int> known[64] = {};
    int n = dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
    if (n > 0) return n;
    if (check_cuda(cudaFuncSetAttribute(efla_seq_kernel<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSqSmem), "cudaFuncSetAttribute(efla_seq_kernel)")) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CS);
    cfg.blockDim = dim3(kSeqThreads);
    cfg.dynamicSmemBytes = kSqSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (check_cuda(cudaOccupancyMaxActiveClusters(&n, efla_seq_kernel<CS>, &cfg), "cudaOccupancyMaxActiveClusters(efla_seq_kernel)")) return 0;
    if (dev < 64 && n > 0) known[dev].store(n, std::memory_order_relaxed);
    return n;
}
}  // namespace

int efla_seq_launch(const EflaParams& p, cudaStream_t stream) {
    int dev = 0;
    const int rc = current_device(&dev);
    if (rc) return rc;
    const int one = resident_clusters<1>(dev), two = resident_clusters<2>(dev), four = resident_clusters<4>(dev);
    if (one <= 0 || two <= 0 || four <= 0) return BNF4_ERR_CUDA;
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
    const int nd = (p.hidden / p.heads + 63) >> 6;
    // Few units leave SMs idle: two or four CTAs share one as long as all units still run at once and every CTA has a block of columns. One head of
    // 512, 32 sequences: 71 us with one, 55 with two, 41 with four; 37 and 70: 71 with one, 55 with two. (Every CTA stages all of K, so sums keep their order;
    // with partial sums over shares of the columns two took 48 and four 39 us, and other bits.) A second pass costs more than sharing gains.
    const int cs = units <= four && nd >= 4 ? 4 : units <= two && nd >= 2 ? 2 : 1;
    const bool early = p.seqs * static_cast<long long>(p.T) * p.hidden <= kPdlStreamElems;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(units * cs));
    cfg.blockDim = dim3(kSeqThreads);
    cfg.dynamicSmemBytes = kSqSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (cs > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = static_cast<unsigned>(cs);
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (early) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, cs == 4 ? efla_seq_kernel<4> : cs == 2 ? efla_seq_kernel<2> : efla_seq_kernel<1>, p);  // errors surface in check_launch
    return check_launch("efla_seq_kernel");
}

}  // namespace bnf4
