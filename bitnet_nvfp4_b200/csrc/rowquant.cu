// Row-wise NVFP4 quantisers and their fused front-ends (bandwidth-bound kernels).
//
// One warp owns one row; lane l owns the 16-element scale blocks l, l+32, ... of that row, so a
// 512-wide int8 row is one coalesced 16-byte load per lane, the e2m1 codes leave as one 8-byte
// store per lane and the four scale bytes of a 64-column group leave as one 32-bit word.
// Every variant produces the same three things the reference's kernels produce -- the int8 copy,
// the packed e2m1 codes and the ue4m3 scale bytes in the tcgen05-friendly atom layout -- and can
// additionally emit the exact int32 projections t[row][v] = sum_k q[row][k] * vec[v][k] that the
// rank-r GEMM epilogue consumes.
//
// Reference semantics restated here (file:line in the reference project):
//   plain int8 rows            src/cuda_kernels.cu:1545-1625   (nvfp4_quantize_a / _b)
//   stacked QKV weights        src/cuda_kernels.cu:2748-2854   (nvfp4_quantize_wqkv_fused)
//   embedding (+dense noise)   src/cuda_kernels.cu:2014-2109
//   embedding (+rank-r noise)  src/cuda_kernels.cu:1360-1389   (element formula of embed_update_lora)
//   + pos, GELU                src/cuda_kernels.cu:2260-2349
//   activation / GELU          src/cuda_kernels.cu:1783-1878, 2500-2589
//   abs-mean norm              src/cuda_kernels.cu:2928-3031
//   residual add + norm        src/cuda_kernels.cu:3033-3143

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace bnf4 {

namespace {

constexpr int kMaxBlocksPerLane = 8;        // rows of up to 32*8*16 = 4096 columns ...
constexpr int kMaxBlocksPerLaneInt8 = 16;  // ... and 8192 for plain int8 rows (weight matrices of wide MLPs)

// Clears the scale bytes of the rows and columns that pad the last atoms, so that callers need not clear the array (a launch of its own).
__device__ __forceinline__ void pad_scales(const RowQuantParams& p) {
    const int nblk = p.cols_out >> 4, k_atoms = sf_k_atoms(p.cols_out), rows_pad = (p.rows + 127) & ~127;
    const int tail = nblk & 3;  // first padding column of the last atom (0: none)
    const int first = tail ? 0 : p.rows;
    const int count = (rows_pad - first) * k_atoms;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const int row = first + i / k_atoms, a = i % k_atoms;
        uint8_t* word = p.out_sf + sf_offset(row, 4 * a, k_atoms);
        if (row >= p.rows) *reinterpret_cast<uint32_t*>(word) = 0u;
        else if (tail && a == k_atoms - 1)
            for (int b = tail; b < 4; ++b) word[b] = 0;
    }
}

template <int FE, int NB>
__global__ void __launch_bounds__(256) rowquant_kernel(const RowQuantParams p, const uint8_t* __restrict__ lut) {
    pdl_trigger();
    const int warps_per_cta = blockDim.x >> 5;
    const int lane = threadIdx.x & 31;
    pdl_wait();
    if (p.pad_sf) pad_scales(p);
    const long long row = static_cast<long long>(blockIdx.x + opaque_zero()) * warps_per_cta + (threadIdx.x >> 5);
    if (row >= p.rows) return;

    const int nblk = p.cols_out >> 4;
    // rows fit 31 bits (p.rows is an int): one 32-bit division instead of a 64-bit division and remainder
    const unsigned urow = static_cast<unsigned>(row);
    const int member = p.rows_per_member > 0 ? static_cast<int>(urow / static_cast<unsigned>(p.rows_per_member)) : 0;
    const int row_in_member = p.rows_per_member > 0 ? static_cast<int>(urow - static_cast<unsigned>(member) * static_cast<unsigned>(p.rows_per_member)) : static_cast<int>(row);
    const int pair = member >> 1;
    const float ns = p.rows_per_member > 0 ? ((member & 1) ? -p.sigma : p.sigma) : p.sigma * static_cast<float>(p.anti_fixed);

    int xw[NB][4];  // stage-1 int8 values of this lane's blocks, four per word
    int sum_abs = 0;

    if constexpr (FE == FE_ADD_ABSMEAN) {
        if (p.zero_t != nullptr && lane < p.zero_n) p.zero_t[static_cast<size_t>(row) * p.zero_n + lane] = 0;
    }

    // ---------------- stage 1: produce integer values ----------------
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int kb = lane + 32 * i;
        xw[i][0] = xw[i][1] = xw[i][2] = xw[i][3] = 0;
        if (kb >= nblk) continue;
        const int k0 = kb << 4;
        int vals[16];
        if constexpr (FE == FE_INT8 || FE == FE_ABSMEAN || FE == FE_WQKV) {
            const int8_t* src;
            if constexpr (FE == FE_WQKV) {
                const int H = p.cols_in;
                const int g = static_cast<int>(row) / H;
                const int rig = static_cast<int>(row) - g * H;
                src = (g == 0 ? p.wq : (g == 1 ? p.wk : (g == 2 ? p.wv : p.wb))) + static_cast<size_t>(g < 3 ? rig : 0) * H;
            } else {
                src = p.in_i8 + static_cast<size_t>(row) * p.ld_in;
            }
            if (p.vec_ok && k0 + 16 <= p.cols_in) {
                const int4 raw = *reinterpret_cast<const int4*>(src + k0);
                const int w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int e = 0; e < 16; ++e) vals[e] = static_cast<int>(static_cast<int8_t>((w[e >> 2] >> (8 * (e & 3))) & 0xff));
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) vals[e] = (k0 + e < p.cols_in) ? static_cast<int>(src[k0 + e]) : 0;
            }
        } else if constexpr (FE == FE_EMBED_DENSE || FE == FE_EMBED_LOWRANK) {
            const int trow = p.row_mod > 0 ? static_cast<int>(urow % static_cast<unsigned>(p.row_mod)) : static_cast<int>(row);
            const int tok = static_cast<int>(p.tokens[static_cast<size_t>(trow) * p.token_stride]);
            const int8_t* e_w = p.emb_w + static_cast<size_t>(tok) * p.cols_in;
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const int j = k0 + e;
                float f = static_cast<float>(e_w[j]);
                if constexpr (FE == FE_EMBED_DENSE) {
                    if (p.emb_noise != nullptr && ns != 0.0f) {
                        const int8_t* e_n = p.emb_noise + static_cast<size_t>(pair) * p.noise_pair_stride + static_cast<size_t>(tok) * p.cols_in;
                        f = fmaf(ns, static_cast<float>(e_n[j]), f);
                    }
                } else {
                    if (ns != 0.0f) {
                        const int8_t* A = p.embA + static_cast<size_t>(pair) * p.embA_pair_stride + static_cast<size_t>(tok) * p.rank;
                        const int8_t* B = p.embB + static_cast<size_t>(pair) * p.embB_pair_stride + j;  // [rank][H]
                        int pert = 0;
                        for (int r = 0; r < p.rank; ++r) pert += static_cast<int>(A[r]) * static_cast<int>(B[static_cast<size_t>(r) * p.cols_in]);
                        f = fmaf(ns * p.c_rank, static_cast<float>(pert), f);
                    }
                }
                vals[e] = clip_int8(rint_to_int(f));
            }
        } else if constexpr (FE == FE_POS_GELU || FE == FE_POS_GELU_ABSMEAN || FE == FE_ACT) {
            size_t in_row = static_cast<size_t>(row);
            if constexpr (FE != FE_ACT) {
                if (p.gather_rows > 0) {  // per-member table of rows indexed by token
                    const unsigned ti = p.row_mod > 0 ? urow % static_cast<unsigned>(p.row_mod) : urow;
                    in_row = static_cast<size_t>(member) * p.gather_rows + p.tokens[static_cast<size_t>(ti) * p.token_stride];
                }
            }
            const float* src = p.in_f32 + in_row * p.ld_in;
            float f[16];
            if (p.vec_ok && k0 + 16 <= p.cols_in) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 v4 = *reinterpret_cast<const float4*>(src + k0 + 4 * q);
                    f[4 * q + 0] = v4.x; f[4 * q + 1] = v4.y; f[4 * q + 2] = v4.z; f[4 * q + 3] = v4.w;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) f[e] = (k0 + e < p.cols_in) ? src[k0 + e] : 0.0f;
            }
            if constexpr (FE == FE_ACT) {
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    float x = f[e];
                    if (p.act_mode == 1) x = x < 0.0f ? 0.0f : x;
                    else if (p.act_mode == 2) x = tanhf(__fdiv_rn(x, 127.0f)) * 127.0f;
                    int qx;
                    if (p.act_mode == 3) qx = gelu_q8(x, p.act_scale);
                    else qx = clip_int8(rint_to_int(x));
                    vals[e] = (k0 + e < p.cols_in) ? qx : 0;
                }
            } else {
                const int prow = p.pos_mod > 0 ? (row_in_member % p.pos_mod) : 0;
                const float* pos = p.pos + static_cast<size_t>(prow) * p.cols_in;
                const int8_t* pn = p.pos_noise != nullptr
                                       ? p.pos_noise + static_cast<size_t>(pair) * p.noise_pair_stride + static_cast<size_t>(prow) * p.cols_in
                                       : nullptr;
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    float pv = pos[k0 + e];
                    if (pn != nullptr) pv = fmaf(ns, static_cast<float>(pn[k0 + e]), pv);
                    vals[e] = gelu_q8(f[e] + pv, p.act_scale);
                }
            }
        } else if constexpr (FE == FE_ADD_ABSMEAN) {
            int8_t* xr = p.inout_i8 + static_cast<size_t>(row) * p.cols_in;
            const float* yr = p.in_f32 + static_cast<size_t>(row) * p.ld_in;
            const int4 raw = *reinterpret_cast<const int4*>(xr + k0);
            const int w[4] = {raw.x, raw.y, raw.z, raw.w};
            int upd[4] = {0, 0, 0, 0};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 y4 = *reinterpret_cast<const float4*>(yr + k0 + 4 * q);
                const float yy[4] = {y4.x, y4.y, y4.z, y4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int old = static_cast<int>(static_cast<int8_t>((w[q] >> (8 * j)) & 0xff));
                    const int v = clip_int8(old + rint_to_int(__fmul_rn(yy[j], p.add_scale)));
                    vals[4 * q + j] = v;
                    upd[q] |= (v & 0xff) << (8 * j);
                }
            }
            *reinterpret_cast<int4*>(xr + k0) = make_int4(upd[0], upd[1], upd[2], upd[3]);
        }
        if constexpr (FE == FE_ABSMEAN || FE == FE_ADD_ABSMEAN || FE == FE_POS_GELU_ABSMEAN) {
#pragma unroll
            for (int e = 0; e < 16; ++e) sum_abs += abs(vals[e]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) xw[i][q] = pack4_i8(vals[4 * q], vals[4 * q + 1], vals[4 * q + 2], vals[4 * q + 3]);
    }

    // ---------------- stage 2: abs-mean normalisation (integer-exact row sum) ----------------
    float inv = 1.0f;
    if constexpr (FE == FE_ABSMEAN || FE == FE_ADD_ABSMEAN || FE == FE_POS_GELU_ABSMEAN) {
        const int total = __reduce_add_sync(0xffffffffu, sum_abs);
        float abs_mean = __fdiv_rn(static_cast<float>(total), static_cast<float>(p.cols_in));
        if (abs_mean < 1.0f) abs_mean = 1.0f;
        inv = __fdiv_rn(p.norm_scale, abs_mean);
    }

    // ---------------- stage 3: emit int8 copy, codes, scales, rank-r projections ----------------
    int tacc[kMaxTVec];
#pragma unroll
    for (int v = 0; v < kMaxTVec; ++v) tacc[v] = 0;

    const int k_atoms = sf_k_atoms(p.cols_out);
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        const int kb = lane + 32 * i;
        const bool active = kb < nblk;
        if (!__any_sync(0xffffffffu, active)) continue;
        const int k0 = kb << 4;
        int w[4] = {0, 0, 0, 0};
        int qi[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) qi[e] = 0;
        if (active) {
            if constexpr (FE == FE_POS_GELU_ABSMEAN) {
                // residual stream = the pre-norm values
                *reinterpret_cast<int4*>(p.inout_i8 + static_cast<size_t>(row) * p.cols_in + k0) =
                    make_int4(xw[i][0], xw[i][1], xw[i][2], xw[i][3]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    int v = static_cast<int>(static_cast<int8_t>((xw[i][q] >> (8 * j)) & 0xff));
                    if constexpr (FE == FE_ABSMEAN || FE == FE_ADD_ABSMEAN || FE == FE_POS_GELU_ABSMEAN)
                        v = clip_int8(rint_to_int(__fmul_rn(static_cast<float>(v), inv)));
                    qi[4 * q + j] = v;
                }
                w[q] = pack4_i8(qi[4 * q], qi[4 * q + 1], qi[4 * q + 2], qi[4 * q + 3]);
            }
            if (p.out_q != nullptr) {
                int8_t* dst = p.out_q + static_cast<size_t>(row) * p.ld_q + k0;
                if (p.vec_ok_q) *reinterpret_cast<int4*>(dst) = make_int4(w[0], w[1], w[2], w[3]);
                else {
#pragma unroll
                    for (int e = 0; e < 16; ++e) dst[e] = static_cast<int8_t>((w[e >> 2] >> (8 * (e & 3))) & 0xff);
                }
            }
        }
        float row_scale = 1.0f;
        if constexpr (FE == FE_WQKV) {
            const int g = static_cast<int>(row) / p.cols_in;
            row_scale = g == 0 ? p.q_scale : (g == 1 ? p.k_scale : (g == 2 ? p.v_scale : p.b_scale));
        }
        uint32_t sfb = 0, lo = 0, hi = 0;
        if (active) {
            if constexpr (FE == FE_WQKV) quant_block16(w, row_scale, true, sfb, lo, hi);
            else quant_block16_lut(qi, lut, sfb, lo, hi);
            *reinterpret_cast<uint2*>(p.out_codes + (static_cast<size_t>(row) * p.cols_out + k0) / 2) = make_uint2(lo, hi);
        }
        // four neighbouring lanes hold the four scale bytes of one 32-bit word of the atom layout
        const int base_lane = lane & ~3;
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) word |= (__shfl_sync(0xffffffffu, sfb, base_lane + j) & 0xffu) << (8 * j);
        if (active && (lane & 3) == 0)
            *reinterpret_cast<uint32_t*>(p.out_sf + sf_offset(static_cast<int>(row), kb, k_atoms)) = word;

        if (p.nvec > 0 && active) {
            const int8_t* tv = p.tvec + static_cast<size_t>(pair) * p.tvec_pair_stride + k0;
#pragma unroll
            for (int v = 0; v < kMaxTVec; ++v) {
                if (v < p.nvec) {
                    const int4 bv = *reinterpret_cast<const int4*>(tv + static_cast<size_t>(v) * p.cols_out);
                    int a = tacc[v];
                    a = __dp4a(w[0], bv.x, a);
                    a = __dp4a(w[1], bv.y, a);
                    a = __dp4a(w[2], bv.z, a);
                    a = __dp4a(w[3], bv.w, a);
                    tacc[v] = a;
                }
            }
        }
    }
    if (p.nvec > 0) {
#pragma unroll
        for (int v = 0; v < kMaxTVec; ++v) {
            if (v < p.nvec) {
                const int tot = __reduce_add_sync(0xffffffffu, tacc[v]);
                if (lane == 0) p.t_out[static_cast<size_t>(row) * p.nvec + v] = tot;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Float-domain fast path for the front-ends the population forward runs once or twice per layer
// (embedding + rank-r noise, + pos / GELU / abs-mean norm, residual add + abs-mean norm, abs-mean norm of int8 rows), and for plain int8
// rows and fp32 activations (16384 x 512 fp32 with one projection: 20.3 us in rowquant_kernel, one row per warp and CTA launch).
//
// Same results as rowquant_kernel, fewer and cheaper instructions: int8 values travel as exact small integers in
// fp32 ("v"), or biased by 1.5 * 2^23 ("t = v + M", whose low byte is the int8), so that
//   * bytes become floats with one byte-permute and one subtraction, and floats become bytes with a byte-permute;
//   * rint() is an addition of M (round-to-nearest-even, like cvt.rni), clip8(rint(x)) = rint(clamp(x, +-127));
//   * the block maximum is a float max; its bit pattern addresses a 1 KB shared-memory table of {1 / scale, scale byte},
//     and the sixteen codes come from the conversion instruction applied to n * (1 / scale) (e2m1x8_table);
// the table is loaded once by a persistent CTA that then walks rows with a grid stride.
// Requirements (checked by the host; otherwise rowquant_kernel runs): 16-byte aligned rows, cols_in == cols_out <= 2048.
// ------------------------------------------------------------------------------------------------
// |b0| + |b1| + |b2| + |b3| of four signed bytes: sum of absolute differences between the bytes offset by 128 and 128
__device__ __forceinline__ uint32_t abs_sum_bytes4(uint32_t w) { return __vsadu4(w ^ 0x80808080u, 0x80808080u); }
__device__ __forceinline__ uint2 lds_u64(uint32_t saddr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(saddr));
    return v;
}
// Eight of a lane's sixteen fp32 values (or its sixteen halves). The lanes' values lie 64 bytes apart, so that a load instruction touches
// sixteen lines whatever its width, and a line is asked for by two or four of them: 32-byte loads halve both. They pass by L1, which the tables'
// lines then keep; 16-byte loads (rows off a 32-byte boundary: wide = false) need their lines there until the last quarter is read, which a
// streaming load does not promise. 16-byte streaming -> 16-byte plain -> 32-byte -> 32-byte past L1, us: fp32 rows in L2, 16384 x 512
// 10.3 -> 9.4 -> 9.0 -> 8.9; + position / GELU 262144 x 512 219 -> 218 -> 191 -> 192, 65536 x 2048 with 16 projections 343 -> 318 -> 304 -> 287.
// FIRST: their lines are the first to leave L2, as a streaming load's are (kFirstToo).
template <bool FIRST = false>
__device__ __forceinline__ void load8(const void* src, bool wide, uint4& a, uint4& b) {
    if (wide && FIRST) {
        asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                     : "l"(src));
    } else if (wide) {
        asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                     : "l"(src));
    } else {
        a = *reinterpret_cast<const uint4*>(src);
        b = *(reinterpret_cast<const uint4*>(src) + 1);
    }
}
__device__ __forceinline__ float4 as_float4(const uint4& v) { return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w)); }
template <bool FIRST = false>
__device__ __forceinline__ void load8(const float* src, bool wide, float4& a, float4& b) {
    uint4 ua, ub;
    load8<FIRST>(static_cast<const void*>(src), wide, ua, ub);
    a = as_float4(ua);
    b = as_float4(ub);
}
// Element ownership as in rowquant_kernel: lane l owns the 16-element scale blocks l, l + 32, ... (NB of them).
// NV = upper bound of p.nvec this instance handles (4 or kMaxTVec): the projection loops carry no tests beyond it.
// BATCH (more than four projections): a 16-byte load per block and vector, one dp4a per four bytes, a warp reduction (8 cycles) per sum and
// sixteen accumulators cost more than the quantisation itself. A warp therefore quantises p.batch consecutive rows, keeping their int8
// values in shared memory, and reads each vector once for all of them. Rows of up to 1024 columns: eight rows, integer matrix instructions
// (vectors as rows of A, staged rows as columns of B: 4096 products in 8 cycles, no reduction over lanes). Wider rows: four rows (eight would
// leave one block per SM), where half of B would be empty; four vectors at a time with dp4a, whose 4 x 4 sums are folded over the warp
// together, are faster there (262144 x 2048, 16 projections: 559 us, 619 us with matrix instructions, 997 us one row at a time).
// 88800 x 320 with eight projections: 80 us one row at a time, 43 us with dp4a on four rows, 34 us here. With four projections (the
// batched driver's instance, 1048576 x 512) one row at a time stays ahead: 337 us against 390 us.
// p.batch is 1 where the rows would not give every resident warp a batch.
__host__ __device__ constexpr int batch_rows(int nb) { return nb >= 4 ? 4 : 8; }
__host__ __device__ constexpr int batch_smem(int nb) { return 8 * batch_rows(nb) * nb * 32 * 16; }
// 16-byte piece c of staged row r: odd rows swap the halves of 128-byte lines, so that two rows' reads share no bank
__device__ __forceinline__ int stage_piece(int r, int c, int nb) { return r * (nb * 32) + (c ^ ((r & 1) << 2)); }

__device__ __forceinline__ void mma_s8_16832(int (&d)[4], int a0, int a1, int a2, int a3, int b0, int b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// t[row0 + r][v] of the rows staged by this warp. Lane (g, tq) supplies 16 contiguous bytes of vectors g and g + 8 and of row g: which of the
// 64 columns of a step meet in which instruction does not matter for the sum, as long as both sides agree.
template <int NB>
__device__ __forceinline__ void project_rows(const RowQuantParams& p, const int4* stage, unsigned row0, unsigned nrows, int nblk, int lane) {
    const int g = lane >> 2, tq = lane & 3;
    const unsigned pair_rows = 2u * static_cast<unsigned>(p.rows_per_member);
    for (unsigned r0 = 0; r0 < nrows;) {  // rows r0 .. r1 - 1 belong to one pair
        const unsigned pair = pair_rows > 0 ? (row0 + r0) / pair_rows : 0u;
        const unsigned r1 = pair_rows > 0 ? min(nrows, (pair + 1u) * pair_rows - row0) : nrows;
        const int8_t* tv = p.tvec + static_cast<size_t>(pair) * p.tvec_pair_stride;
        if constexpr (NB >= 4) {
            constexpr int R = batch_rows(NB);
            for (int v0 = 0; v0 < p.nvec; v0 += 4) {
                int acc[R][4];
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[r][j] = 0;
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    if (lane + 32 * i >= nblk) continue;
                    int4 b[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j)  // the last group may be short: its tail repeats the last vector and is not stored
                        b[j] = *reinterpret_cast<const int4*>(tv + 16 * lane + static_cast<size_t>(min(v0 + j, p.nvec - 1)) * p.cols_out + 512 * i);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int4 w = stage[stage_piece(r, lane + 32 * i, NB)];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            int a = acc[r][j];
                            a = __dp4a(w.x, b[j].x, a);
                            a = __dp4a(w.y, b[j].y, a);
                            a = __dp4a(w.z, b[j].z, a);
                            acc[r][j] = __dp4a(w.w, b[j].w, a);
                        }
                    }
                }
                // sixteen sums over 32 lanes: lane l ends with the sum of value l / 2 (row l / 8, vector (l / 2) % 4)
                int x[8], y[4], z[2];
                const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4, h2 = lane & 2;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int lo = acc[q >> 2][q & 3], hi = acc[2 + (q >> 2)][q & 3];
                    x[q] = (h16 ? hi : lo) + __shfl_xor_sync(0xffffffffu, h16 ? lo : hi, 16);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) y[q] = (h8 ? x[4 + q] : x[q]) + __shfl_xor_sync(0xffffffffu, h8 ? x[q] : x[4 + q], 8);
#pragma unroll
                for (int q = 0; q < 2; ++q) z[q] = (h4 ? y[2 + q] : y[q]) + __shfl_xor_sync(0xffffffffu, h4 ? y[q] : y[2 + q], 4);
                int tot = (h2 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, h2 ? z[0] : z[1], 2);
                tot += __shfl_xor_sync(0xffffffffu, tot, 1);
                const unsigned r = lane >> 3;
                const int v = v0 + ((lane >> 1) & 3);
                if (!(lane & 1) && r >= r0 && r < r1 && v < p.nvec) p.t_out[static_cast<size_t>(row0 + r) * p.nvec + v] = tot;
            }
        } else {
            const int8_t* tg = tv + static_cast<size_t>(g) * p.cols_out + 16 * tq;
            int d[4] = {0, 0, 0, 0}, d2[4] = {0, 0, 0, 0};  // two chains
#pragma unroll 4
            for (int c0 = 0; c0 < nblk; c0 += 4) {
                int4 lo = make_int4(0, 0, 0, 0), hi = lo, w = lo;
                if (c0 + tq < nblk) {
                    if (g < p.nvec) lo = *reinterpret_cast<const int4*>(tg + 16 * c0);
                    if (g + 8 < p.nvec) hi = *reinterpret_cast<const int4*>(tg + 8 * static_cast<size_t>(p.cols_out) + 16 * c0);
                    if (g < batch_rows(NB)) w = stage[stage_piece(g, c0 + tq, NB)];
                }
                mma_s8_16832(d, lo.x, hi.x, lo.y, hi.y, w.x, w.y);
                mma_s8_16832(d2, lo.z, hi.z, lo.w, hi.w, w.z, w.w);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const unsigned r = 2 * tq + (e & 1);
                const int v = g + 8 * (e >> 1);
                if (r >= r0 && r < r1 && v < p.nvec) p.t_out[static_cast<size_t>(row0 + r) * p.nvec + v] = d[e] + d2[e];
            }
        }
        r0 = r1;
    }
}

// Which instances keep a row's bytes, not its sixteen floats per block, until the norm is known, and how many blocks of them share an SM.
// Rows of more than 512 columns hold 32 or 64 floats a lane: with them in registers too few warps are resident to cover the latency of the
// loads, without them the bytes are widened a second time. 65536 rows, us:
//   floats kept -> bytes kept, 2 / 3 blocks an SM: int8 rows, 2048 columns, 16 projections 153 -> 136 / 140, 4 projections 126 -> 99 / 100,
//     1024 columns 55 -> 53 / 52; + position / GELU, 1024 columns 137 -> 122 / 124, 2048 columns, 16 projections 344 -> 347 / 393;
//     + branch, 1024 columns, 1 projection 67 -> 70 / 71, 2048 columns, 4 projections 160 -> 165 / 148, but 4000 such rows 17.8 -> 19.6
//   floats kept, 2 / 3 blocks: + position / GELU, 2048 columns, 4 projections 257 / 261 (one block: 294, with 16-byte loads).
//     fp32 rows past 1024 columns stay at one block: three take 65536 x 2048 from 186 to 154, but 4000 x 1984 from 16 to 20.
// 1500 / 4000 / 16384 / 65536 rows behind another kernel: 2048 bytes 6.3 -> 5.9, 9.5 -> 8.7, 28 -> 20, 95 -> 68; 768 + position / GELU 8.5 -> 8.0, 13.6 -> 12.1,
// 37.5 -> 33.7, 135 -> 109. Dearer: launches of 1000 to 2300 rows behind one another (4.5 -> 4.8, 6.6 -> 7.0: the next launch starts in the room that the smaller register
// count leaves), and + position / GELU with four projections 200 rows 7.7 -> 8.0, 4700 x 1024 from DRAM 15.2 -> 16.9 (from L2 14.8 both).
template <int FE, int NB, int NV>
constexpr bool kKeepBytes = NB > 1 && (FE == FE_ABSMEAN || (FE == FE_POS_GELU_ABSMEAN && NB <= 2));
template <int FE, int NB, int NV>
constexpr int kFastCtas = NB <= 1 ? 4 : kKeepBytes<FE, NB, NV> ? 2 : (NB <= 2 || NV > 4 || FE == FE_POS_GELU_ABSMEAN) ? 2 : 1;

// Rows that are read once leave L2 first, or they push out what is read again (the residual stream, the codes). 16-byte streaming loads -> 32-byte -> 32-byte, first to leave, us:
//   halves, + branch: 65536 x 512 29.4 -> 31.1 -> 28.9, 32000 x 1024 34.8 -> 36.8 -> 32.6, 1048576 x 512 455 -> 450 -> 450;
//   fp32 rows, activation, from DRAM: 16384 x 512 10.7 -> 10.7 -> 10.5, with four projections 12.4 -> 13.2 -> 12.0, 8000 x 512 with four 8.2 -> 9.1 -> 7.9; from L2 16384 x 512
//     10.5 -> 9.9 -> 9.9, two buffers in turn 10.8 -> 9.9 -> 10.7; a GEMM behind 16384 x 512 that are new each time 21.8 -> 20.8 for both.
// fp32 rows of the residual add have instances of their own for it, FIRST, from 40 to 128 MB (L2 holds 126): 32000 x 512 20.4 -> 21.5 -> 19.0, 12000 x 1024 17.1 -> 19.6 -> 16.6,
// 65536 x 512 35.4 -> 38.3 -> 33.3; but 262144 x 512 149 -> 140 -> 162.
template <int FE, int NB>
constexpr bool kFirstToo = FE == FE_ADD_ABSMEAN && NB <= 2;

// MODEL: powers of two for rows per member, columns and positions, 32-byte aligned rows, one or four projections: no test or division for any of it
// (the 32-byte rule: 262144 x 512 + position / GELU 198 -> 191 us).
// ZERO: the MODEL instance that also clears p.zero_t, for launches of up to kPdlStreamElems elements; larger ones have a memset in front (the test
// and the store cost the default model's instance 4 %, 0.6 of 14.4 ms a step, the memsets 0.1 ms).
template <int FE, int NB, int NV, bool MODEL = false, bool ZERO = !MODEL, bool FIRST = false>
__global__ void __launch_bounds__(256, kFastCtas<FE, NB, NV>) rowquant_fast_kernel(const RowQuantParams p, const uint8_t* __restrict__ lut) {
    pdl_trigger();
    __shared__ __align__(16) uint2 tab_s[128];  // per amax: {bits of fl(1 / scale), scale byte}
    if (threadIdx.x < 128) tab_s[threadIdx.x] = __ldg(reinterpret_cast<const uint2*>(lut + kQuantBlockTabOffset) + threadIdx.x);
    __syncthreads();
    pdl_wait();  // the table is constant; the rows are the predecessor's
    if (!MODEL && p.pad_sf) pad_scales(p);
    // entry address from the bit pattern of (amax + kRoundBias): (bits - kRoundBiasBits) * 8, folded into one constant
    const uint32_t tab_c = static_cast<uint32_t>(__cvta_generic_to_shared(tab_s)) - (static_cast<uint32_t>(kRoundBiasBits) << 3);
    const float M = kRoundBias;
    constexpr bool kNorm = (FE == FE_ADD_ABSMEAN || FE == FE_POS_GELU_ABSMEAN || FE == FE_ABSMEAN);
    constexpr bool PACK = kKeepBytes<FE, NB, NV>;
    const float gelu_safe = gelu_q8_safe(p.act_scale);
    const bool wide = MODEL || p.wide_ok;

    const int lane = threadIdx.x & 31;
    const int nblk = p.cols_out >> 4;
    const int k_atoms = sf_k_atoms(p.cols_out);
    const unsigned rows = static_cast<unsigned>(p.rows);
    const bool cols_pow2 = MODEL || (p.cols_in & (p.cols_in - 1)) == 0;
    // token / position indices wrap at powers of two in every model configuration: masks instead of divisions per row
    const bool row_mod_pow2 = MODEL || (p.row_mod > 0 && (p.row_mod & (p.row_mod - 1)) == 0);
    const bool pos_mod_pow2 = MODEL || (p.pos_mod > 0 && (p.pos_mod & (p.pos_mod - 1)) == 0);
    const int rpm_shift = (p.rows_per_member > 0 && (p.rows_per_member & (p.rows_per_member - 1)) == 0) ? __ffs(p.rows_per_member) - 1 : -1;
    const float inv_cols = 1.0f / static_cast<float>(p.cols_in);
    constexpr bool BATCH = NV > 4;
    const unsigned batch = BATCH ? static_cast<unsigned>(p.batch) : 1u;
    int4* stage = nullptr;
    if constexpr (BATCH) {
        extern __shared__ __align__(16) int4 batch_stage[];
        stage = batch_stage + (threadIdx.x >> 5) * (batch_rows(NB) * NB * 32);
    }
    unsigned in_batch = 0;  // rows of the current batch before this one
    unsigned next_row;
    for (unsigned row = ((blockIdx.x + opaque_zero()) * 8u + (threadIdx.x >> 5)) * batch; row < rows; row = next_row) {
        next_row = BATCH && in_batch + 1 < batch ? row + 1 : row - in_batch + gridDim.x * 8u * batch;
        // rows per member is a power of two in every model configuration: a shift instead of a division per row
        const int member = (MODEL || p.rows_per_member > 0) ? static_cast<int>((MODEL || rpm_shift >= 0) ? row >> rpm_shift : row / static_cast<unsigned>(p.rows_per_member)) : 0;
        const int row_in_member = (MODEL || p.rows_per_member > 0) ? static_cast<int>(row - static_cast<unsigned>(member) * static_cast<unsigned>(p.rows_per_member)) : static_cast<int>(row);
        const int pair = member >> 1;
        const float ns = (MODEL || p.rows_per_member > 0) ? ((member & 1) ? -p.sigma : p.sigma) : p.sigma * static_cast<float>(p.anti_fixed);

        // The row this warp takes next starts its trip from DRAM to L2 now: a warp holds one row's loads at a time, too few
        // bytes in flight to cover the DRAM latency with the narrow inputs (int8 rows, a branch travelling as halves).
        if constexpr (FE == FE_ADD_ABSMEAN || FE == FE_ABSMEAN) {
            if (next_row < rows) {
#pragma unroll
                for (int i = 0; i < NB; ++i) {
                    const int k0 = (lane + 32 * i) << 4;
                    if (k0 >= p.cols_in) continue;
                    if constexpr (FE == FE_ABSMEAN) {
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.in_i8 + static_cast<size_t>(next_row) * p.ld_in + k0));
                    } else if (MODEL || p.in_f16) {
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.inout_i8 + static_cast<size_t>(next_row) * p.cols_in + k0));
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const __half*>(p.in_f32) + static_cast<size_t>(next_row) * p.ld_in + k0));
                    }
                }
            }
        }

        if constexpr (FE == FE_ADD_ABSMEAN && ZERO) {
            if (p.zero_t != nullptr && lane < p.zero_n) p.zero_t[static_cast<size_t>(row) * p.zero_n + lane] = 0;
        }

        // ---------------- stage 1: integer values of the row as floats ----------------
        float vf[PACK ? 1 : NB][16];
        uint32_t raw_w[FE == FE_INT8 || PACK ? NB : 1][4];  // the row's bytes (FE_INT8, PACK)
        uint32_t sum_abs = 0;  // sum of |value| over this lane's elements (exact integer)
        int tok = 0;
        float a_r[4] = {0.f, 0.f, 0.f, 0.f};
        if constexpr (FE == FE_EMBED_LOWRANK) {
            const int trow = p.row_mod > 0 ? static_cast<int>(row_mod_pow2 ? row & static_cast<unsigned>(p.row_mod - 1) : row % static_cast<unsigned>(p.row_mod)) : static_cast<int>(row);
            tok = static_cast<int>(p.tokens[static_cast<size_t>(trow) * p.token_stride]);
            if (ns != 0.0f) {
                const int8_t* A = p.embA + static_cast<size_t>(pair) * p.embA_pair_stride + static_cast<size_t>(tok) * p.rank;
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (r < p.rank) a_r[r] = static_cast<float>(A[r]);
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int kb = lane + 32 * i;
            const int k0 = kb << 4;
            if (kb >= nblk) {
                if constexpr (!PACK) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) vf[i][e] = 0.0f;
                }
                continue;
            }
            if constexpr (FE == FE_INT8) {
                const int4 raw = *reinterpret_cast<const int4*>(p.in_i8 + static_cast<size_t>(row) * p.ld_in + k0);
                const uint32_t rw[4] = {static_cast<uint32_t>(raw.x), static_cast<uint32_t>(raw.y), static_cast<uint32_t>(raw.z), static_cast<uint32_t>(raw.w)};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    raw_w[i][q] = rw[q];  // the int8 copy and the projections take the bytes as they are
                    bytes4_to_float(rw[q], &vf[i][4 * q]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) vf[i][4 * q + j] = fmaxf(vf[i][4 * q + j], -127.0f);  // -128 is quantised as -127
                }
            } else if constexpr (FE == FE_ACT) {
                const float* src = p.in_f32 + static_cast<size_t>(row) * p.ld_in + k0;
                float4 f4[4];
#pragma unroll
                for (int q = 0; q < 4; q += 2) {
                    if constexpr (NB >= 2) {  // streaming loads suit these: 65536 x 1024 71.8 us, 74.0 with the 32-byte ones; 4000 x 1984 from DRAM 16.0, 19.5
                        f4[q] = __ldcs(reinterpret_cast<const float4*>(src) + q);
                        f4[q + 1] = __ldcs(reinterpret_cast<const float4*>(src) + q + 1);
                    } else {
                        load8<true>(src + 4 * q, wide, f4[q], f4[q + 1]);
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float x[4] = {f4[q].x, f4[q].y, f4[q].z, f4[q].w};
                    if (p.act_mode == 3) {
                        float tb[4];
                        gelu_q8x4(x, p.act_scale, gelu_safe, tb);
#pragma unroll
                        for (int j = 0; j < 4; ++j) vf[i][4 * q + j] = tb[j] - M;
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            float y = x[j];
                            if (p.act_mode == 1) y = y < 0.0f ? 0.0f : y;
                            else if (p.act_mode == 2) y = tanhf(__fdiv_rn(y, 127.0f)) * 127.0f;
                            const float r = (fminf(fmaxf(y, -127.0f), 127.0f) + M) - M;  // clip8(rint(y))
                            vf[i][4 * q + j] = y != y ? 0.0f : r;                        // (an integer conversion turns NaN into 0)
                        }
                    }
                }
            } else if constexpr (FE == FE_ABSMEAN) {
                const int4 raw = *reinterpret_cast<const int4*>(p.in_i8 + static_cast<size_t>(row) * p.ld_in + k0);
                const uint32_t rw[4] = {static_cast<uint32_t>(raw.x), static_cast<uint32_t>(raw.y), static_cast<uint32_t>(raw.z), static_cast<uint32_t>(raw.w)};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if constexpr (PACK) raw_w[i][q] = rw[q];
                    else bytes4_to_float(rw[q], &vf[i][4 * q]);
                    sum_abs += abs_sum_bytes4(rw[q]);
                }
            } else if constexpr (FE == FE_ADD_ABSMEAN) {
                int8_t* xr = p.inout_i8 + static_cast<size_t>(row) * p.cols_in;
                const float* yr = p.in_f32 + static_cast<size_t>(row) * p.ld_in;
                const int4 raw = *reinterpret_cast<const int4*>(xr + k0);
                const uint32_t rw[4] = {static_cast<uint32_t>(raw.x), static_cast<uint32_t>(raw.y), static_cast<uint32_t>(raw.z), static_cast<uint32_t>(raw.w)};
                float4 y4[4];
                if (MODEL || p.in_f16) {  // the branch output as IEEE halves (exact widening)
                    const uint4* yh = reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(p.in_f32) + static_cast<size_t>(row) * p.ld_in + k0);
                    uint4 h0, h1;
                    if constexpr (NB > 2) {  // (as below)
                        h0 = __ldcs(yh);
                        h1 = __ldcs(yh + 1);
                    } else {
                        load8<true>(yh, wide, h0, h1);
                    }
                    const uint32_t hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&hw[2 * q])), hi = __half22float2(*reinterpret_cast<const __half2*>(&hw[2 * q + 1]));
                        y4[q] = make_float4(lo.x, lo.y, hi.x, hi.y);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q += 2) {
                        if constexpr (NB > 2) {  // streaming loads: 4000 x 2048 from DRAM 14.9 us, 15.3 with the 32-byte ones (halves, 4 projections: 17.8, 20.6)
                            y4[q] = __ldcs(reinterpret_cast<const float4*>(yr + k0 + 4 * q));
                            y4[q + 1] = __ldcs(reinterpret_cast<const float4*>(yr + k0 + 4 * q) + 1);
                        } else {
                            load8<FIRST>(yr + k0 + 4 * q, wide, y4[q], y4[q + 1]);
                        }
                    }
                }
                uint32_t upd[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float yy[4] = {y4[q].x, y4[q].y, y4[q].z, y4[q].w};
                    float oldf[4], tb[4];
                    bytes4_to_float(rw[q], oldf);
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        // old + rint(y * add_scale), clipped to +-127, all on biased floats: resid_add_biased on packed fp32 pairs
                        // (each half rounds like the scalar instruction)
                        const float2 tr = __fadd2_rn(__fmul2_rn(make_float2(yy[j], yy[j + 1]), make_float2(p.add_scale, p.add_scale)), make_float2(M, M));
                        const float2 sm = __fadd2_rn(tr, make_float2(oldf[j], oldf[j + 1]));
                        tb[j] = fminf(fmaxf(sm.x, M - 127.0f), M + 127.0f);
                        tb[j + 1] = fminf(fmaxf(sm.y, M - 127.0f), M + 127.0f);
                        if constexpr (!PACK) {
                            const float2 vv = __fadd2_rn(make_float2(tb[j], tb[j + 1]), make_float2(-M, -M));
                            vf[i][4 * q + j] = vv.x;
                            vf[i][4 * q + j + 1] = vv.y;
                        }
                    }
                    upd[q] = biased4_to_bytes(tb[0], tb[1], tb[2], tb[3]);
                    if constexpr (PACK) raw_w[i][q] = upd[q];
                    sum_abs += abs_sum_bytes4(upd[q]);
                }
                *reinterpret_cast<int4*>(xr + k0) = make_int4(static_cast<int>(upd[0]), static_cast<int>(upd[1]), static_cast<int>(upd[2]), static_cast<int>(upd[3]));
            } else if constexpr (FE == FE_POS_GELU_ABSMEAN) {
                size_t in_row = static_cast<size_t>(row);
                if (p.gather_rows > 0) {  // per-member table of rows indexed by token
                    const unsigned ti = p.row_mod > 0 ? (row_mod_pow2 ? row & static_cast<unsigned>(p.row_mod - 1) : row % static_cast<unsigned>(p.row_mod)) : row;
                    in_row = static_cast<size_t>(member) * p.gather_rows + p.tokens[static_cast<size_t>(ti) * p.token_stride];
                }
                const float* src = p.in_f32 + in_row * p.ld_in;
                const int prow = p.pos_mod > 0 ? (pos_mod_pow2 ? row_in_member & (p.pos_mod - 1) : row_in_member % p.pos_mod) : 0;
                const float* pos = p.pos + static_cast<size_t>(prow) * p.cols_in;
                uint32_t pw[4] = {0x0u, 0x0u, 0x0u, 0x0u};
                const bool has_pn = p.pos_noise != nullptr;
                if (has_pn) {
                    const int4 pn = *reinterpret_cast<const int4*>(p.pos_noise + static_cast<size_t>(pair) * p.noise_pair_stride + static_cast<size_t>(prow) * p.cols_in + k0);
                    pw[0] = static_cast<uint32_t>(pn.x); pw[1] = static_cast<uint32_t>(pn.y); pw[2] = static_cast<uint32_t>(pn.z); pw[3] = static_cast<uint32_t>(pn.w);
                }
                float4 f4[4];
#pragma unroll
                for (int q = 0; q < 4; q += 2) load8(src + k0 + 4 * q, wide, f4[q], f4[q + 1]);
                float4 pos4[2];
                uint32_t resid[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (!(q & 1)) load8(pos + k0 + 4 * q, wide, pos4[0], pos4[1]);
                    const float4 p4 = pos4[q & 1];
                    const float ff[4] = {f4[q].x, f4[q].y, f4[q].z, f4[q].w};
                    float pv[4] = {p4.x, p4.y, p4.z, p4.w};
                    if (has_pn) {
                        float pnf[4];
                        bytes4_to_float(pw[q], pnf);
#pragma unroll
                        for (int j = 0; j < 4; ++j) pv[j] = fmaf(ns, pnf[j], pv[j]);
                    }
                    float x[4], tb[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[j] = ff[j] + pv[j];
                    gelu_q8x4(x, p.act_scale, gelu_safe, tb);
                    if constexpr (!PACK) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) vf[i][4 * q + j] = tb[j] - M;
                    }
                    resid[q] = biased4_to_bytes(tb[0], tb[1], tb[2], tb[3]);
                    if constexpr (PACK) raw_w[i][q] = resid[q];
                    sum_abs += abs_sum_bytes4(resid[q]);
                }
                // residual stream = the pre-norm values
                *reinterpret_cast<int4*>(p.inout_i8 + static_cast<size_t>(row) * p.cols_in + k0) =
                    make_int4(static_cast<int>(resid[0]), static_cast<int>(resid[1]), static_cast<int>(resid[2]), static_cast<int>(resid[3]));
            } else {  // FE_EMBED_LOWRANK
                const int4 ew = *reinterpret_cast<const int4*>(p.emb_w + static_cast<size_t>(tok) * p.cols_in + k0);
                const uint32_t eww[4] = {static_cast<uint32_t>(ew.x), static_cast<uint32_t>(ew.y), static_cast<uint32_t>(ew.z), static_cast<uint32_t>(ew.w)};
                float pert[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) pert[e] = 0.0f;
                if (ns != 0.0f) {
                    const int8_t* B = p.embB + static_cast<size_t>(pair) * p.embB_pair_stride + k0;  // [rank][H]
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (r < p.rank) {
                            const int4 bw = *reinterpret_cast<const int4*>(B + static_cast<size_t>(r) * p.cols_in);
                            const uint32_t bww[4] = {static_cast<uint32_t>(bw.x), static_cast<uint32_t>(bw.y), static_cast<uint32_t>(bw.z), static_cast<uint32_t>(bw.w)};
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                float bf[4];
                                bytes4_to_float(bww[q], bf);
#pragma unroll
                                for (int j = 0; j < 4; ++j) pert[4 * q + j] = fmaf(a_r[r], bf[j], pert[4 * q + j]);  // exact: small integers
                            }
                        }
                    }
                }
                const float nsc = ns * p.c_rank;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    float wf[4];
                    bytes4_to_float(eww[q], wf);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float f = ns != 0.0f ? fmaf(nsc, pert[4 * q + j], wf[j]) : wf[j];
                        vf[i][4 * q + j] = (fminf(fmaxf(f, -127.0f), 127.0f) + M) - M;  // clip8(rint(f))
                    }
                }
            }
        }

        // ---------------- stage 2: abs-mean normalisation (integer-exact row sum) ----------------
        float inv = 1.0f;
        if constexpr (kNorm) {
            const int total = static_cast<int>(__reduce_add_sync(0xffffffffu, sum_abs));
            // a power-of-two column count divides exactly by multiplication
            float abs_mean = cols_pow2 ? __fmul_rn(static_cast<float>(total), inv_cols) : __fdiv_rn(static_cast<float>(total), static_cast<float>(p.cols_in));
            if (abs_mean < 1.0f) abs_mean = 1.0f;
            inv = __fdiv_rn(p.norm_scale, abs_mean);
        }

        // ---------------- stage 3: int8 copy, codes, scales, rank-r projections ----------------
        int tacc[BATCH ? 1 : NV];
#pragma unroll
        for (int v = 0; v < (BATCH ? 1 : NV); ++v) tacc[v] = 0;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int kb = lane + 32 * i;
            const bool active = kb < nblk;
            if (!__any_sync(0xffffffffu, active)) continue;
            const int k0 = kb << 4;
            uint32_t w[4] = {0u, 0u, 0u, 0u};
            uint32_t sfb = 0;
            if (active) {
                float tq[16];
                float am = 0.0f;
                float un[16];
                const float* v16 = un;
                if constexpr (PACK) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) bytes4_to_float(raw_w[i][q], un + 4 * q);
                } else {
                    v16 = vf[i];
                }
                if (kNorm && inv > 1.0f) {  // same for the whole row; only then can |v| * inv pass 127
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        const float n = fminf(fmaxf(__fmul_rn(v16[e], inv), -127.0f), 127.0f);
                        am = fmaxf(am, fabsf(n));
                        tq[e] = n + M;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 16; e += 2) {  // packed fp32 pairs: each half rounds like the scalar instruction
                        float2 n = make_float2(v16[e], v16[e + 1]);
                        if constexpr (kNorm) n = __fmul2_rn(n, make_float2(inv, inv));
                        am = fmax3(am, fabsf(n.x), fabsf(n.y));
                        const float2 t2 = __fadd2_rn(n, make_float2(M, M));
                        tq[e] = t2.x;
                        tq[e + 1] = t2.y;
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if constexpr (FE == FE_INT8) w[q] = raw_w[i][q];
                    else w[q] = biased4_to_bytes(tq[4 * q], tq[4 * q + 1], tq[4 * q + 2], tq[4 * q + 3]);
                }
                if (!MODEL && p.out_q != nullptr)
                    *reinterpret_cast<int4*>(p.out_q + static_cast<size_t>(row) * p.ld_q + k0) =
                        make_int4(static_cast<int>(w[0]), static_cast<int>(w[1]), static_cast<int>(w[2]), static_cast<int>(w[3]));
                const uint2 ent = lds_u64((__float_as_uint(am + M) << 3) + tab_c);
                sfb = ent.y;
                const float rs = __uint_as_float(ent.x);
                uint32_t lo, hi;
                if constexpr (kNorm) {
                    lo = e2m1x8_biased(tq, rs);
                    hi = e2m1x8_biased(tq + 8, rs);
                } else {  // the values are integers already
                    lo = e2m1x8_table(v16, rs);
                    hi = e2m1x8_table(v16 + 8, rs);
                }
                *reinterpret_cast<uint2*>(p.out_codes + (static_cast<size_t>(row) * p.cols_out + k0) / 2) = make_uint2(lo, hi);
            }
            // one byte per lane: four neighbouring lanes fill one 32-bit word of the atom layout, the warp touches the same
            // eight sectors a word store would
            if (active) p.out_sf[sf_offset(static_cast<int>(row), kb, k_atoms)] = static_cast<uint8_t>(sfb);

            if constexpr (BATCH) {
                if (active)
                    stage[stage_piece(static_cast<int>(in_batch), kb, NB)] =
                        make_int4(static_cast<int>(w[0]), static_cast<int>(w[1]), static_cast<int>(w[2]), static_cast<int>(w[3]));
            } else if constexpr (MODEL) {
                if (active) {
                    const int8_t* tv = p.tvec + static_cast<size_t>(pair) * p.tvec_pair_stride + k0;
#pragma unroll
                    for (int v = 0; v < NV; ++v) {
                        const int4 bv = *reinterpret_cast<const int4*>(tv + static_cast<size_t>(v) * p.cols_out);
                        int a = tacc[v];
                        a = __dp4a(static_cast<int>(w[0]), bv.x, a);
                        a = __dp4a(static_cast<int>(w[1]), bv.y, a);
                        a = __dp4a(static_cast<int>(w[2]), bv.z, a);
                        a = __dp4a(static_cast<int>(w[3]), bv.w, a);
                        tacc[v] = a;
                    }
                }
            } else if (p.nvec > 0 && active) {
                const int8_t* tv = p.tvec + static_cast<size_t>(pair) * p.tvec_pair_stride + k0;
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    if (v < p.nvec) {
                        const int4 bv = *reinterpret_cast<const int4*>(tv + static_cast<size_t>(v) * p.cols_out);
                        int a = tacc[v];
                        a = __dp4a(static_cast<int>(w[0]), bv.x, a);
                        a = __dp4a(static_cast<int>(w[1]), bv.y, a);
                        a = __dp4a(static_cast<int>(w[2]), bv.z, a);
                        a = __dp4a(static_cast<int>(w[3]), bv.w, a);
                        tacc[v] = a;
                    }
                }
            }
        }
        if constexpr (BATCH) {
            if (in_batch + 1 == batch || row + 1 == rows) {
                __syncwarp();
                project_rows<NB>(p, stage, row - in_batch, in_batch + 1, nblk, lane);
                if (row + 1 == rows) break;
                __syncwarp();
                in_batch = 0;
            } else {
                ++in_batch;
            }
        } else if constexpr (MODEL) {
            if constexpr (NV == 4) {
                const int t0 = __reduce_add_sync(0xffffffffu, tacc[0]), t1 = __reduce_add_sync(0xffffffffu, tacc[1]);
                const int t2 = __reduce_add_sync(0xffffffffu, tacc[2]), t3 = __reduce_add_sync(0xffffffffu, tacc[3]);
                if (lane == 0) *reinterpret_cast<int4*>(p.t_out + static_cast<size_t>(row) * 4) = make_int4(t0, t1, t2, t3);
            } else {
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const int tot = __reduce_add_sync(0xffffffffu, tacc[v]);
                    if (lane == 0) p.t_out[static_cast<size_t>(row) * NV + v] = tot;
                }
            }
        } else if (p.nvec > 0) {
            if (p.nvec == 4 && (reinterpret_cast<uintptr_t>(p.t_out) & 15) == 0) {  // the four column groups of the fused q | k | v | beta projection: one 16-byte store
                const int t0 = __reduce_add_sync(0xffffffffu, tacc[0]), t1 = __reduce_add_sync(0xffffffffu, tacc[1]);
                const int t2 = __reduce_add_sync(0xffffffffu, tacc[2]), t3 = __reduce_add_sync(0xffffffffu, tacc[3]);
                if (lane == 0) *reinterpret_cast<int4*>(p.t_out + static_cast<size_t>(row) * 4) = make_int4(t0, t1, t2, t3);
            } else {
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    if (v < p.nvec) {
                        const int tot = __reduce_add_sync(0xffffffffu, tacc[v]);
                        if (lane == 0) p.t_out[static_cast<size_t>(row) * p.nvec + v] = tot;
                    }
                }
            }
        }
    }
}

// CTAs of a fast-kernel instance that fit one SM, per device (0 = not looked up yet)
template <int FE, int NB, int NV, bool MODEL = false, bool ZERO = !MODEL, bool FIRST = false>
std::atomic<int> resident_ctas[64] = {};

template <int FE>
int launch(const RowQuantParams& p, cudaStream_t stream) {
    if (p.rows <= 0 || p.cols_out <= 0) return BNF4_OK;
    if ((p.cols_out & 15) != 0) return set_error(BNF4_ERR_INVALID, "rowquant: cols_out=%d must be a multiple of 16", p.cols_out);
    constexpr int max_cols = 32 * 16 * (FE == FE_INT8 ? kMaxBlocksPerLaneInt8 : kMaxBlocksPerLane);
    if (p.cols_out > max_cols) return set_error(BNF4_ERR_INVALID, "rowquant: cols_out=%d exceeds %d", p.cols_out, max_cols);
    if (p.nvec > kMaxTVec) return set_error(BNF4_ERR_INVALID, "rowquant: nvec=%d exceeds %d", p.nvec, kMaxTVec);
    if (p.out_codes == nullptr || p.out_sf == nullptr) return set_error(BNF4_ERR_INVALID, "rowquant: null output");
    if ((reinterpret_cast<uintptr_t>(p.out_codes) & 7) || (reinterpret_cast<uintptr_t>(p.out_sf) & 3))
        return set_error(BNF4_ERR_INVALID, "rowquant: outputs must be 8-byte (codes) / 4-byte (scales) aligned");
    const int warps = 8;
    const unsigned ctas = static_cast<unsigned>((static_cast<long long>(p.rows) + warps - 1) / warps);
    const int nblk = p.cols_out >> 4;
    const uint8_t* lut = get_quant_lut();
    if (lut == nullptr) return BNF4_ERR_CUDA;
    const bool early = static_cast<long long>(p.rows) * p.cols_out <= kPdlStreamElems;
    if constexpr (FE == FE_EMBED_LOWRANK || FE == FE_POS_GELU_ABSMEAN || FE == FE_ADD_ABSMEAN || FE == FE_ABSMEAN || FE == FE_ACT || FE == FE_INT8) {
        auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
        bool fast = p.cols_in == p.cols_out && nblk <= 128 && (p.out_q == nullptr || p.vec_ok_q) && al16(p.inout_i8 ? p.inout_i8 : nullptr);
        if (FE == FE_ABSMEAN || FE == FE_INT8) fast = fast && p.vec_ok && p.in_i8 != nullptr;
        if (FE == FE_ACT) fast = fast && p.vec_ok && p.in_f32 != nullptr;
        if (FE == FE_ADD_ABSMEAN) fast = fast && al16(p.in_f32) && (p.ld_in % (p.in_f16 ? 8 : 4)) == 0;
        if (FE == FE_ADD_ABSMEAN && p.in_f16 && !fast) return set_error(BNF4_ERR_INVALID, "rowquant: fp16 input needs 16-byte aligned rows and cols_in == cols_out <= 2048");
        if (FE == FE_POS_GELU_ABSMEAN)
            fast = fast && p.vec_ok && al16(p.pos) && (p.pos_noise == nullptr || (al16(p.pos_noise) && (p.noise_pair_stride % 16) == 0));
        if (FE == FE_EMBED_LOWRANK)
            fast = fast && al16(p.emb_w) && p.rank >= 0 && p.rank <= 4 && (p.sigma == 0.0f || (al16(p.embB) && (p.embB_pair_stride % 16) == 0));
        if (fast) {
            int dev = 0;
            int rc = current_device(&dev);
            if (rc) return rc;
            const int sms = multiprocessors(dev);
            if (sms <= 0) return BNF4_ERR_CUDA;
            // persistent CTAs: exactly as many as are resident at once (each loads its 1 KB copy of the table once)
            auto run = [&](auto kernel, std::atomic<int>* resident, int smem = 0, int batch = 1) -> int {
                int per_sm = resident[dev].load(std::memory_order_relaxed);
                if (per_sm == 0) {  // looked up once per kernel and device
                    int rc2 = smem > 48 * 1024 ? check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "cudaFuncSetAttribute(rowquant_fast_kernel)") : BNF4_OK;
                    if (!rc2) rc2 = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem), "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
                    if (rc2) return rc2;
                    per_sm = std::max(per_sm, 1);
                    resident[dev].store(per_sm, std::memory_order_relaxed);
                }
                unsigned work = ctas;
                const unsigned fit = static_cast<unsigned>(sms) * static_cast<unsigned>(per_sm);
                RowQuantParams q = p;
                q.batch = 1;
                if (batch > 1 && ctas >= batch * fit) {  // a batch of rows for every resident warp
                    q.batch = batch;
                    work = (ctas + batch - 1) / batch;
                }
                launch_pdl_if(early, kernel, std::min(work, fit), warps * 32, smem, stream, q, lut);
                return BNF4_OK;
            };
            // the batched driver's calls at hidden <= 512: see MODEL above
            auto pow2 = [](long long v) { return v > 0 && (v & (v - 1)) == 0; };
            bool model = p.wide_ok && nblk <= 32 && (FE == FE_ADD_ABSMEAN || FE == FE_ABSMEAN || FE == FE_POS_GELU_ABSMEAN) && pow2(p.cols_in) && pow2(p.rows_per_member) &&
                         p.out_q == nullptr && (p.nvec == 1 || p.nvec == 4) && p.tvec != nullptr && p.t_out != nullptr && al16(p.t_out);
            if (FE == FE_ADD_ABSMEAN) model = model && p.in_f16 != 0;
            if (FE == FE_POS_GELU_ABSMEAN) model = model && pow2(p.pos_mod) && (p.gather_rows <= 0 || pow2(p.row_mod));
            if constexpr (FE == FE_ADD_ABSMEAN || FE == FE_ABSMEAN || FE == FE_POS_GELU_ABSMEAN) {
                if constexpr (FE == FE_ADD_ABSMEAN) {
                    if (model && p.zero_t != nullptr) {
                        rc = p.nvec == 1 ? run(rowquant_fast_kernel<FE, 1, 1, true, true>, resident_ctas<FE, 1, 1, true, true>)
                                         : run(rowquant_fast_kernel<FE, 1, 4, true, true>, resident_ctas<FE, 1, 4, true, true>);
                        if (rc) return rc;
                        return check_launch("rowquant_fast_kernel");
                    }
                }
                if (model) {
                    rc = p.nvec == 1 ? run(rowquant_fast_kernel<FE, 1, 1, true>, resident_ctas<FE, 1, 1, true>) : run(rowquant_fast_kernel<FE, 1, 4, true>, resident_ctas<FE, 1, 4, true>);
                    if (rc) return rc;
                    return check_launch("rowquant_fast_kernel");
                }
            }
            const long long row_bytes = 4LL * p.rows * p.cols_out;
            const bool first = !p.in_f16 && row_bytes >= (40LL << 20) && row_bytes <= (128LL << 20);  // (kFirstToo)
            auto run_nv = [&](auto nb, auto nv) -> int {
                constexpr int NB = decltype(nb)::value, NV = decltype(nv)::value;
                constexpr int smem = NV > 4 ? batch_smem(NB) : 0, batch = NV > 4 ? batch_rows(NB) : 1;
                if constexpr (kFirstToo<FE, NB>) {
                    if (first) return run(rowquant_fast_kernel<FE, NB, NV, false, true, true>, resident_ctas<FE, NB, NV, false, true, true>, smem, batch);
                }
                return run(rowquant_fast_kernel<FE, NB, NV>, resident_ctas<FE, NB, NV>, smem, batch);
            };
            auto run_nb = [&](auto nb) -> int { return p.nvec <= 4 ? run_nv(nb, std::integral_constant<int, 4>()) : run_nv(nb, std::integral_constant<int, kMaxTVec>()); };
            rc = nblk <= 32 ? run_nb(std::integral_constant<int, 1>()) : nblk <= 64 ? run_nb(std::integral_constant<int, 2>()) : run_nb(std::integral_constant<int, 4>());
            if (rc) return rc;
            return check_launch("rowquant_fast_kernel");
        }
    }
    if (nblk <= 32) launch_pdl_if(early, rowquant_kernel<FE, 1>, ctas, warps * 32, 0, stream, p, lut);
    else if (nblk <= 64) launch_pdl_if(early, rowquant_kernel<FE, 2>, ctas, warps * 32, 0, stream, p, lut);
    else if (nblk <= 128) launch_pdl_if(early, rowquant_kernel<FE, 4>, ctas, warps * 32, 0, stream, p, lut);
    else if (nblk <= 256) launch_pdl_if(early, rowquant_kernel<FE, 8>, ctas, warps * 32, 0, stream, p, lut);
    else {
        if constexpr (FE == FE_INT8) launch_pdl_if(early, rowquant_kernel<FE, 16>, ctas, warps * 32, 0, stream, p, lut);
    }
    return check_launch("rowquant_kernel");
}

bool aligned16(const void* ptr, long long ld_bytes) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && (ld_bytes & 15) == 0; }

}  // namespace

int rowquant_dispatch(int fe, RowQuantParams p, cudaStream_t stream) {
    // vectorised access is a property of the caller's pointers and strides; decided once on the host
    switch (fe) {
        case FE_INT8: case FE_ABSMEAN:
            p.vec_ok = aligned16(p.in_i8, p.ld_in) ? 1 : 0; break;
        case FE_WQKV:
            p.vec_ok = (aligned16(p.wq, p.cols_in) && aligned16(p.wk, p.cols_in) && aligned16(p.wv, p.cols_in) && aligned16(p.wb, p.cols_in)) ? 1 : 0; break;
        case FE_POS_GELU: case FE_POS_GELU_ABSMEAN: case FE_ACT:
            p.vec_ok = aligned16(p.in_f32, static_cast<long long>(p.ld_in) * 4) ? 1 : 0; break;
        default: p.vec_ok = 1; break;
    }
    // 32-byte loads: fp32 rows (or halves), and the position table's
    const long long in_bytes = p.in_f16 ? 2 : 4;
    p.wide_ok = (reinterpret_cast<uintptr_t>(p.in_f32) & 31) == 0 && ((p.ld_in * in_bytes) & 31) == 0 &&
                (fe != FE_POS_GELU_ABSMEAN || ((reinterpret_cast<uintptr_t>(p.pos) & 31) == 0 && (p.cols_in & 7) == 0));
    p.vec_ok_q = (p.out_q != nullptr && aligned16(p.out_q, p.ld_q)) ? 1 : 0;
    if (fe == FE_ADD_ABSMEAN || fe == FE_POS_GELU_ABSMEAN) {
        if (!aligned16(p.inout_i8, p.cols_in))
            return set_error(BNF4_ERR_INVALID, "rowquant: residual stream must be 16-byte aligned with hidden %% 16 == 0");
    }
    if (p.in_f16 && fe != FE_ADD_ABSMEAN) return set_error(BNF4_ERR_INVALID, "rowquant: fp16 input is supported by the residual-add front-end only");
    if (fe == FE_ADD_ABSMEAN && !aligned16(p.in_f32, static_cast<long long>(p.ld_in) * (p.in_f16 ? 2 : 4)))
        return set_error(BNF4_ERR_INVALID, "rowquant: fp32 input must be 16-byte aligned");
    if ((fe == FE_POS_GELU || fe == FE_POS_GELU_ABSMEAN || fe == FE_EMBED_DENSE || fe == FE_EMBED_LOWRANK || fe == FE_ADD_ABSMEAN || fe == FE_ABSMEAN) &&
        p.cols_in != p.cols_out)
        return set_error(BNF4_ERR_INVALID, "rowquant: this front-end needs cols_in == cols_out");
    if (p.nvec > 0 && !aligned16(p.tvec, p.cols_out)) return set_error(BNF4_ERR_INVALID, "rowquant: projection vectors must be 16-byte aligned");
    if (p.gather_rows > 0 && ((fe != FE_POS_GELU && fe != FE_POS_GELU_ABSMEAN) || p.tokens == nullptr || p.rows_per_member <= 0))
        return set_error(BNF4_ERR_INVALID, "rowquant: gather_rows needs a pos+GELU front-end, tokens and rows_per_member");
    if (fe == FE_ADD_ABSMEAN && p.zero_t != nullptr && p.rows > 0 && static_cast<long long>(p.rows) * p.cols_out > kPdlStreamElems) {
        const int rc = check_cuda(cudaMemsetAsync(p.zero_t, 0, static_cast<size_t>(p.rows) * p.zero_n * sizeof(int32_t), stream), "cudaMemsetAsync(projections)");
        if (rc) return rc;
        p.zero_t = nullptr;
    }
    switch (fe) {
        case FE_INT8: return launch<FE_INT8>(p, stream);
        case FE_WQKV: return launch<FE_WQKV>(p, stream);
        case FE_EMBED_DENSE: return launch<FE_EMBED_DENSE>(p, stream);
        case FE_EMBED_LOWRANK: return launch<FE_EMBED_LOWRANK>(p, stream);
        case FE_POS_GELU: return launch<FE_POS_GELU>(p, stream);
        case FE_POS_GELU_ABSMEAN: return launch<FE_POS_GELU_ABSMEAN>(p, stream);
        case FE_ACT: return launch<FE_ACT>(p, stream);
        case FE_ABSMEAN: return launch<FE_ABSMEAN>(p, stream);
        case FE_ADD_ABSMEAN: return launch<FE_ADD_ABSMEAN>(p, stream);
    }
    return set_error(BNF4_ERR_INVALID, "rowquant: unknown front-end %d", fe);
}

}  // namespace bnf4
