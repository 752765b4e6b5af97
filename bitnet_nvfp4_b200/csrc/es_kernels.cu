// Cross-entropy fitness, counter-hash noise and the ES weight update (bandwidth / integer-pipe kernels).
//
// Reference semantics restated here (file:line in the reference project):
//   cross entropy          src/efla_lm_kernels.cu:252-311
//   noise fill             src/efla_lm_kernels.cu:73-86, 352-385
//   pair seeds             src/efla_lm_kernels.cu:1844-1852
//   Z and sum of squares   src/efla_lm_kernels.cu:1854-1890
//   inv_rms                src/efla_lm_kernels.cu:2003-2021
//   shadow update          src/efla_lm_kernels.cu:1892-1922
// All reductions run in a fixed order so that every rank of a data-parallel job computes identical bits
// (the reference uses unordered float atomics).

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace bnf4 {

namespace {

// ------------------------------------------------------------------------------------------------
// Cross entropy. One warp per row; lane l holds logits l, l+32, ...
// ------------------------------------------------------------------------------------------------
constexpr int kCeMaxPerLane = 32;  // vocab <= 1024

__device__ __forceinline__ float ce_row_loss(const float* lg, const float* bias, const float* noise_f, const int8_t* noise_i,
                                             float bns, int vocab, int y, int lane) {
    float v[kCeMaxPerLane];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < kCeMaxPerLane; ++j) {
        const int i = lane + 32 * j;
        if (i < vocab) {
            float x = lg[i];
            if (bias != nullptr) x += bias[i];
            if (noise_f != nullptr) x = fmaf(bns, noise_f[i], x);
            if (noise_i != nullptr) x = fmaf(bns, static_cast<float>(noise_i[i]), x);
            v[j] = x;
            mx = fmaxf(mx, x);
        } else {
            v[j] = -INFINITY;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < kCeMaxPerLane; ++j) {
        const int i = lane + 32 * j;
        if (i < vocab) sum += expf(v[j] - mx);
    }
    sum = warp_sum_f(sum);
    // the target's value lives in lane y%32, slot y/32
    float vy = 0.0f;
#pragma unroll
    for (int j = 0; j < kCeMaxPerLane; ++j)
        if (j == (y >> 5)) vy = v[j];
    vy = __shfl_sync(0xffffffffu, vy, y & 31);
    return -(vy - mx - logf(sum + 1e-9f));
}

// API form: a single CTA sums the rows of one token step in a fixed order and adds the total to *loss_accum.
__global__ void __launch_bounds__(1024) ce_step_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                                                      const float* __restrict__ bias_noise, float bns,
                                                      const uint8_t* __restrict__ targets_t, int token_stride, int vocab, int batch,
                                                      float* loss_accum) {
    pdl_wait();
    after(logits, bias, bias_noise, targets_t);
    __shared__ float part[32];  // a warp per row: 32 rows, the reference driver's batch, in one go
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float acc = 0.0f;
    for (int b = warp; b < batch; b += 32) {
        const int y = static_cast<int>(targets_t[static_cast<size_t>(b) * token_stride]);
        acc += ce_row_loss(logits + static_cast<size_t>(b) * vocab, bias, bias_noise, nullptr, bns, vocab, y, lane);
    }
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < 32; ++w) t += part[w];
        loss_accum[0] += t;
    }
}

// Population form. A member's rows form 16 groups of consecutive rows, a group eight chains: chain w adds rows w, w + 8, .. of its group in
// order, the group adds its chains in order, the mean adds the groups in double. Every loss is a function of the logits alone: grid and
// member count only say which warps compute the row losses. (1024 pairs rank losses that differ in the last place: another order of these
// sums moves some across each other and with them the update.)
// Grid (16 split, members), split 1, 2, 4 or 8: `split` blocks share a group, `split` warps a chain. Member counters (zero before the launch, zero
// again after it): the member's last block forms the mean; without them split is 1, partial[member * 16 + group] holds the groups'
// sums and ce_finalize_kernel follows. With split > 1 partial holds the chains' sums, 128 per member.
constexpr int kCeChunks = 16;
// SHARED false: the instance for split 1 (with the split as a variable a full wave of the default model, 1048576 rows, took 484 instead of 397 us).
template <bool SHARED>
struct CeRows {
    int split, r0, r1, chain, j;  // this warp: rows r0 + chain + 8 (j + split k) below r1
    __device__ explicit CeRows(int rows_per_member) {
        const int warp = threadIdx.x >> 5, per = (rows_per_member + kCeChunks - 1) / kCeChunks;
        split = SHARED ? static_cast<int>(gridDim.x) / kCeChunks : 1;
        const int group = static_cast<int>(blockIdx.x) / split, sub = static_cast<int>(blockIdx.x) - group * split;
        r0 = group * per;
        r1 = min(rows_per_member, r0 + per);
        chain = sub * (8 / split) + warp / split;
        j = warp % split;
    }
    __device__ int row(int k) const { return r0 + chain + 8 * (SHARED ? j + split * k : k); }
    // whether a pass over rows row(k0), .. has any (of this warp; SHARED: of the block, which passes together)
    __device__ bool more(int k0) const { return SHARED ? r0 + 8 * split * k0 < r1 : row(k0) < r1; }
};
// adds the row losses l[i] of rows row(k0 + i) to the chain's sum (kept by its first warp)
template <bool SHARED, int RPI>
__device__ __forceinline__ void ce_add(const CeRows<SHARED>& rr, int pass, const float (&l)[RPI], float& acc) {
    if constexpr (!SHARED) {
#pragma unroll
        for (int i = 0; i < RPI; ++i) acc += l[i];
        return;
    }
    __shared__ float rows[2][8][RPI];
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int i = 0; i < RPI; ++i) rows[pass & 1][warp][i] = l[i];
    __syncthreads();
    if (rr.j == 0)
#pragma unroll
        for (int i = 0; i < RPI; ++i)
            for (int q = 0; q < rr.split; ++q) acc += rows[pass & 1][warp + q][i];
}
template <bool SHARED>
__device__ __forceinline__ void ce_finish(const CeRows<SHARED>& rr, float acc, float* partial, unsigned* counters, int rows_per_member, float* loss_mean) {
    __shared__ float part[8];
    __shared__ bool last;
    const int member = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0 && rr.j == 0) part[warp / rr.split] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        if constexpr (!SHARED) {
            float t = 0.0f;
            for (int w = 0; w < 8; ++w) t += part[w];
            partial[member * kCeChunks + blockIdx.x] = t;
        } else {
            const int chains = 8 / rr.split;
            for (int w = 0; w < chains; ++w) partial[member * (8 * kCeChunks) + blockIdx.x * chains + w] = part[w];
        }
        last = false;
        if (counters != nullptr) {
            __threadfence();
            last = atomicInc(counters + member, gridDim.x - 1) == gridDim.x - 1;  // wraps to zero
        }
    }
    if (counters == nullptr) return;
    __syncthreads();
    if (!last || threadIdx.x >= 32) return;
    __threadfence();
    float group = 0.0f;
    if (lane < kCeChunks) {
        if (!SHARED) group = __ldcg(partial + member * kCeChunks + lane);
        else
            for (int w = 0; w < 8; ++w) group += __ldcg(partial + member * (8 * kCeChunks) + 8 * lane + w);
    }
    double t = static_cast<double>(group);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) loss_mean[member] = static_cast<float>(t / static_cast<double>(rows_per_member));
}
template <bool SHARED>
__global__ void __launch_bounds__(256) ce_population_kernel(const float* __restrict__ logits, int ld, const float* __restrict__ bias,
                                                            const int8_t* __restrict__ bias_noise, float sigma,
                                                            const uint8_t* __restrict__ targets, int vocab, int rows_per_member,
                                                            float* partial, unsigned* counters, float* loss_mean) {
    pdl_wait();
    after(logits, bias, bias_noise, targets);
    const CeRows<SHARED> rr(rows_per_member);
    const int lane = threadIdx.x & 31, member = blockIdx.y;
    const float bns = (member & 1) ? -sigma : sigma;
    const int8_t* nz = bias_noise != nullptr ? bias_noise + static_cast<size_t>(member >> 1) * vocab : nullptr;
    float acc = 0.0f;
    for (int k = 0; rr.more(k); ++k) {
        const int r = rr.row(k);
        float l[1] = {0.0f};
        if (r < rr.r1)
            l[0] = ce_row_loss(logits + (static_cast<size_t>(member) * rows_per_member + r) * ld, bias, nullptr, nz, bns, vocab, static_cast<int>(targets[r]), lane);
        ce_add<SHARED, 1>(rr, k, l, acc);
    }
    ce_finish(rr, acc, partial, counters, rows_per_member, loss_mean);
}

// Streaming form of the same reduction for 16-byte aligned rows and vocab % 4 == 0: lane l owns the float4 groups
// l, l + 32, ... of a row (NV4 groups), the member's bias and noise stay in registers for all rows, and RPI rows are in
// flight per warp so that the load latency of one row hides behind the reductions of the others. The warps walk the
// rows in the same order and add the row losses in the same order as ce_population_kernel.
template <int NV4, int RPI, bool SHARED>
__global__ void __launch_bounds__(256) ce_population_vec_kernel(const float* __restrict__ logits, int ld, const float* __restrict__ bias,
                                                                const int8_t* __restrict__ bias_noise, float sigma,
                                                                const uint8_t* __restrict__ targets, int vocab, int rows_per_member,
                                                                float* partial, unsigned* counters, float* loss_mean) {
    pdl_wait();
    after(logits, bias, bias_noise, targets);
    const CeRows<SHARED> rr(rows_per_member);
    const int lane = threadIdx.x & 31, member = blockIdx.y, r1 = rr.r1;
    const float bns = (member & 1) ? -sigma : sigma;
    const int groups = vocab >> 2;
    float4 bv[NV4], nv[NV4];
#pragma unroll
    for (int j = 0; j < NV4; ++j) {
        const int gi = lane + 32 * j;
        bv[j] = nv[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (gi < groups) {
            if (bias != nullptr) bv[j] = *reinterpret_cast<const float4*>(bias + 4 * gi);
            if (bias_noise != nullptr) {
                const char4 c = *reinterpret_cast<const char4*>(bias_noise + static_cast<size_t>(member >> 1) * vocab + 4 * gi);
                nv[j] = make_float4(static_cast<float>(c.x), static_cast<float>(c.y), static_cast<float>(c.z), static_cast<float>(c.w));
            }
        }
    }
    float acc = 0.0f;
    for (int pass = 0; rr.more(pass * RPI); ++pass) {
        float l[RPI];
        float4 x[RPI][NV4];
        int y[RPI];
#pragma unroll
        for (int i = 0; i < RPI; ++i) {
            const int r = rr.row(pass * RPI + i);
            y[i] = r < r1 ? static_cast<int>(targets[r]) : 0;
            const float* lg = logits + (static_cast<size_t>(member) * rows_per_member + min(r, r1 - 1)) * ld;
#pragma unroll
            for (int j = 0; j < NV4; ++j) {
                const int gi = lane + 32 * j;
                x[i][j] = gi < groups ? __ldcs(reinterpret_cast<const float4*>(lg) + gi) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            }
        }
#pragma unroll
        for (int i = 0; i < RPI; ++i) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < NV4; ++j) {
                if (lane + 32 * j < groups) {  // (x + bias) + bns * noise, like the scalar kernel (zero bias / noise when absent)
                    x[i][j].x = fmaf(bns, nv[j].x, x[i][j].x + bv[j].x);
                    x[i][j].y = fmaf(bns, nv[j].y, x[i][j].y + bv[j].y);
                    x[i][j].z = fmaf(bns, nv[j].z, x[i][j].z + bv[j].z);
                    x[i][j].w = fmaf(bns, nv[j].w, x[i][j].w + bv[j].w);
                }
                mx = fmaxf(fmaxf(mx, fmaxf(x[i][j].x, x[i][j].y)), fmaxf(x[i][j].z, x[i][j].w));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < NV4; ++j) sum += (expf(x[i][j].x - mx) + expf(x[i][j].y - mx)) + (expf(x[i][j].z - mx) + expf(x[i][j].w - mx));
            sum = warp_sum_f(sum);
            // the target's logit is re-read (one broadcast load per row) and perturbed with the same two operations
            const int r = min(rr.row(pass * RPI + i), r1 - 1);
            float vy = logits[(static_cast<size_t>(member) * rows_per_member + r) * ld + y[i]];
            if (bias != nullptr) vy += bias[y[i]];
            if (bias_noise != nullptr) vy = fmaf(bns, static_cast<float>(bias_noise[static_cast<size_t>(member >> 1) * vocab + y[i]]), vy);
            l[i] = rr.row(pass * RPI + i) < r1 ? -(vy - mx - logf(sum + 1e-9f)) : 0.0f;
        }
        ce_add<SHARED, RPI>(rr, pass, l, acc);
    }
    ce_finish(rr, acc, partial, counters, rows_per_member, loss_mean);
}

__global__ void ce_finalize_kernel(const float* __restrict__ partial, int members, int rows_per_member, float* __restrict__ loss_mean) {
    pdl_wait();
    after(partial);
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= members) return;
    double t = 0.0;
    for (int c = 0; c < kCeChunks; ++c) t += static_cast<double>(partial[m * kCeChunks + c]);
    loss_mean[m] = static_cast<float>(t / static_cast<double>(rows_per_member));
}

// ------------------------------------------------------------------------------------------------
// Noise
// ------------------------------------------------------------------------------------------------
__global__ void fill_noise_kernel(int8_t* __restrict__ out, size_t n, uint64_t seed, int use_clt, int clt_k) {
    pdl_wait();
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx < n) out[idx] = static_cast<int8_t>(use_clt != 0 && clt_k == 4 ? noise_clt4(noise_seed(seed), idx) : noise_hash(seed, idx, use_clt != 0, clt_k));
}
__global__ void fill_noise_batched_kernel(const bnf4_noise_desc* __restrict__ descs, int num_desc, int use_clt, int clt_k) {
    pdl_wait();
    after(descs);
    const int di = blockIdx.y;
    if (di >= num_desc) return;
    const bnf4_noise_desc d = descs[di];
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx < d.n)
        d.out[idx] = static_cast<int8_t>(use_clt != 0 && clt_k == 4 ? noise_clt4(noise_seed(d.seed), idx) : noise_hash(d.seed, idx, use_clt != 0, clt_k));
}
__global__ void fill_float_noise_kernel(float* __restrict__ out, int n, uint64_t seed, int use_clt, int clt_k) {
    pdl_wait();
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < n) out[idx] = static_cast<float>(noise_hash(seed, static_cast<uint64_t>(idx), use_clt != 0, clt_k));
}
__global__ void pair_seeds_kernel(uint64_t base_seed, uint64_t epoch, int pairs, uint64_t* __restrict__ out) {
    pdl_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < pairs) out[p] = mix_u64(base_seed, mix_u64(epoch, static_cast<uint64_t>(p)));
}

// ------------------------------------------------------------------------------------------------
// ES update
// ------------------------------------------------------------------------------------------------
__global__ void init_shadow_kernel(const int8_t* __restrict__ w, float* __restrict__ shadow, int n) {
    pdl_wait();
    after(w);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) shadow[i] = static_cast<float>(w[i]);
}

// Z for the dense (full-matrix noise) form; 256 threads per block, one element each.
// idx: the element's index in the whole vector, which keys the hash.
// CLT4: the noise every model uses (sum of four ternary draws).
template <bool CLT4>
__device__ __forceinline__ void z_dense_block(const float* pair_weights, const uint64_t* pair_seeds, uint64_t salt, int pairs, int idx, bool active,
                                              int use_clt, int clt_k, float* out) {
    __shared__ NoiseSeed seeds[256];
    __shared__ float wts[256];
    float z = 0.0f;
    for (int p0 = 0; p0 < pairs; p0 += 256) {
        __syncthreads();
        if (p0 + threadIdx.x < pairs) {
            seeds[threadIdx.x] = noise_seed(mix_u64(pair_seeds[p0 + threadIdx.x], salt));
            wts[threadIdx.x] = pair_weights[p0 + threadIdx.x];
        }
        __syncthreads();
        const int cnt = min(256, pairs - p0);
        if (active) {
            // independent hash chains in flight; the multiply-adds stay in pair order (pairs of weight zero are skipped, like in the
            // reference)
            auto noise = [&](int p) {
                return static_cast<float>(CLT4 ? noise_clt4(seeds[p], static_cast<uint64_t>(idx)) : noise_hash(seeds[p].a, static_cast<uint64_t>(idx), use_clt != 0, clt_k));
            };
            int p = 0;
            for (; p + 4 <= cnt; p += 4) {
                float e[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) e[q] = noise(p + q);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float w = wts[p + q];
                    if (w != 0.0f) z = fmaf(w, e[q], z);
                }
            }
            for (; p < cnt; ++p) {
                const float w = wts[p];
                if (w != 0.0f) z = fmaf(w, noise(p), z);
            }
        }
    }
    if (active) *out = z;
}
template <bool CLT4>
__global__ void __launch_bounds__(256) z_dense_kernel(const float* __restrict__ pair_weights, const uint64_t* __restrict__ pair_seeds,
                                                      uint64_t salt, int pairs, int n, int use_clt, int clt_k, float* __restrict__ Z) {
    pdl_wait();
    after(pair_weights, pair_seeds);
    const int i = blockIdx.x * 256 + threadIdx.x;
    z_dense_block<CLT4>(pair_weights, pair_seeds, salt, pairs, i, i < n, use_clt, clt_k, Z + i);
}
// The same for a table of tensors (the fp32 vectors of a model; in the dense mode also its matrices) in one launch: block b finds
// its tensor by walking the table. With nshards > 1 a tensor that is computed in shards covers this shard's elements only.
template <bool CLT4>
__global__ void __launch_bounds__(256) z_dense_table_kernel(const float* __restrict__ pair_weights, const uint64_t* __restrict__ pair_seeds,
                                                            const ZDenseDesc* __restrict__ descs, int ndesc, int pairs, int use_clt, int clt_k, int shard,
                                                            int nshards, float* __restrict__ z_all) {
    pdl_wait();
    after(pair_weights, pair_seeds);
    int block = static_cast<int>(blockIdx.x), idx0 = 0, n = 0;
    ZDenseDesc d = {};
    for (int t = 0; t < ndesc; ++t) {
        d = descs[t];
        z_dense_range(d, shard, nshards, idx0, n);
        const int blocks = (n + 255) / 256;
        if (block < blocks) break;
        block -= blocks;
    }
    const int i = block * 256 + threadIdx.x;
    z_dense_block<CLT4>(pair_weights, pair_seeds, d.salt, pairs, idx0 + i, i < n, use_clt, clt_k, z_all + d.zoff + idx0 + i);
}

// Rank-r form of Z: Z[i][j] = cscale * sum_p w_p * (sum_r A[p][i][r] * B[p][r][j]), pairs in ascending order with one fused
// multiply-add per pair (reference: src/efla_lm_kernels.cu:1854-1890 applied to the factored noise). The inner sum is a
// small integer, so it is formed exactly in fp32 from factors converted once while they are staged in shared memory.
//
// One launch covers a table of matrices (all ternary matrices of a model): block b locates its matrix and its
// 32-row x 64-column tile by walking the table. Thread (ty, tx) of the 8 x 16 thread tile keeps a 4 x 4 block of Z in
// registers, so one pair costs three shared-memory loads (weight, 4 values of A, 4 of B) for 32 arithmetic
// instructions; factors arrive in chunks of PC pairs, the next chunk's global loads in flight while the current one is
// consumed (registers -> the other shared-memory buffer, one barrier per chunk). With nshards > 1 a matrix whose rows
// divide by nshards is computed only for the rows of this shard.
constexpr int kZTileRows = 32, kZTileCols = 64, kZThreads = 128;

__device__ __forceinline__ void z_shard_rows(int rows, int shard, int nshards, int& r0, int& nr) {
    r0 = 0;
    nr = rows;
    if (nshards > 1 && rows >= nshards && (rows % nshards) == 0) { nr = rows / nshards; r0 = shard * nr; }
}

// The first `table_blocks` blocks compute the tensors whose noise lies in memory as [pair][n] bytes (the step's fp32 vectors): one byte per
// pair and element instead of one hash, same values, same order. They are few and latency-bound, so they start first.
__device__ __forceinline__ void z_table_block(const float* __restrict__ pair_weights, const ZDenseDesc* __restrict__ descs, int ndesc, int block, int pairs, int shard,
                                              int nshards, float* __restrict__ z_all) {
    int idx0 = 0, n = 0;
    ZDenseDesc d = {};
    for (int t = 0; t < ndesc; ++t) {
        d = descs[t];
        z_dense_range(d, shard, nshards, idx0, n);
        const int blocks = (n + kZThreads - 1) / kZThreads;
        if (block < blocks) break;
        block -= blocks;
    }
    const int i = block * kZThreads + static_cast<int>(threadIdx.x);
    if (i >= n) return;
    const int8_t* src = d.noise + idx0 + i;
    float z = 0.0f;
    int p = 0;
    for (; p + 16 <= pairs; p += 16) {
        int8_t e[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) e[q] = src[static_cast<size_t>(p + q) * d.n];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const float w = pair_weights[p + q];
            if (w != 0.0f) z = fmaf(w, static_cast<float>(e[q]), z);
        }
    }
    for (; p < pairs; ++p) {
        const float w = pair_weights[p];
        if (w != 0.0f) z = fmaf(w, static_cast<float>(src[static_cast<size_t>(p) * d.n]), z);
    }
    z_all[d.zoff + idx0 + i] = z;
}

template <int RANK>
__global__ void __launch_bounds__(kZThreads) z_lowrank_tiles_kernel(const float* __restrict__ pair_weights, const ZLowrankDesc* __restrict__ descs,
                                                                    int ndesc, const ZLowrankDesc single, int pairs, float cscale, int shard,
                                                                    int nshards, const ZTables tables) {
    pdl_wait();
    after(pair_weights);
    constexpr int PC = RANK <= 2 ? 16 : 8;  // pairs per chunk
    constexpr int TR = kZTileRows, TC = kZTileCols;
    constexpr int A_PER_THREAD = PC * TR * RANK / kZThreads;        // bytes of A per thread and chunk
    constexpr int B_PER_THREAD = PC * RANK * (TC / 4) / kZThreads;  // 4-byte words of B per thread and chunk
    __shared__ __align__(16) float a_sh[2][PC][RANK][TR];
    __shared__ __align__(16) float b_sh[2][PC][RANK][TC];
    __shared__ float w_sh[2][PC];

    if (static_cast<int>(blockIdx.x) < tables.blocks) {
        z_table_block(pair_weights, tables.descs, tables.ndesc, static_cast<int>(blockIdx.x), pairs, shard, nshards, tables.z_all);
        return;
    }
    // which matrix, which tile
    ZLowrankDesc d = single;
    int tile = static_cast<int>(blockIdx.x) - tables.blocks;
    int r0 = 0, nr = d.rows;
    if (ndesc > 0 && nshards == 1) {
        int lo = 0, hi = ndesc - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (descs[mid].tile0 <= tile) lo = mid; else hi = mid - 1;
        }
        d = descs[lo];
        tile -= d.tile0;
        nr = d.rows;
    } else if (ndesc > 0) {
        int i = 0;
        for (;;) {
            d = descs[i];
            z_shard_rows(d.rows, shard, nshards, r0, nr);
            const int tiles = ((nr + TR - 1) / TR) * ((d.cols + TC - 1) / TC);
            if (tile < tiles) break;
            tile -= tiles;
            if (++i >= ndesc) return;
        }
    }
    const int tiles_x = (d.cols + TC - 1) / TC;
    const int by = tile / tiles_x, bx = tile - by * tiles_x;
    const int row_base = r0 + by * TR, row_end = r0 + nr, col_base = bx * TC;
    const int tid = static_cast<int>(threadIdx.x), ty = tid >> 4, tx = tid & 15;
    const bool b_words = ((reinterpret_cast<uintptr_t>(d.B) & 3) == 0) && ((d.B_ps & 3) == 0) && ((d.cols & 3) == 0);

    int a_raw[A_PER_THREAD];
    uint32_t b_raw[B_PER_THREAD];
    float w_raw = 0.0f;
    auto fetch = [&](int p0) {
#pragma unroll
        for (int k = 0; k < A_PER_THREAD; ++k) {
            const int e = tid + k * kZThreads;
            const int pp = e / (TR * RANK), rem = e - pp * (TR * RANK);  // rem = row * RANK + r: contiguous in A
            const int row = row_base + rem / RANK;
            a_raw[k] = (p0 + pp < pairs && row < row_end) ? static_cast<int>(d.A[static_cast<size_t>(p0 + pp) * d.A_ps + static_cast<size_t>(row_base) * RANK + rem]) : 0;
        }
#pragma unroll
        for (int k = 0; k < B_PER_THREAD; ++k) {
            const int e = tid + k * kZThreads;
            const int pp = e / (RANK * (TC / 4)), rem = e - pp * (RANK * (TC / 4)), r = rem / (TC / 4), c = (rem - r * (TC / 4)) * 4;
            const int col = col_base + c;
            uint32_t v = 0;
            if (p0 + pp < pairs && col < d.cols) {
                const int8_t* src = d.B + static_cast<size_t>(p0 + pp) * d.B_ps + static_cast<size_t>(r) * d.cols + col;
                if (b_words) {
                    v = *reinterpret_cast<const uint32_t*>(src);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (col + q < d.cols) v |= (static_cast<uint32_t>(static_cast<uint8_t>(src[q]))) << (8 * q);
                }
            }
            b_raw[k] = v;
        }
        if (tid < PC) w_raw = (p0 + tid < pairs) ? pair_weights[p0 + tid] : 0.0f;
    };
    auto stage = [&](int buf) {
#pragma unroll
        for (int k = 0; k < A_PER_THREAD; ++k) {
            const int e = tid + k * kZThreads;
            const int pp = e / (TR * RANK), rem = e - pp * (TR * RANK);
            a_sh[buf][pp][rem % RANK][rem / RANK] = static_cast<float>(a_raw[k]);
        }
#pragma unroll
        for (int k = 0; k < B_PER_THREAD; ++k) {
            const int e = tid + k * kZThreads;
            const int pp = e / (RANK * (TC / 4)), rem = e - pp * (RANK * (TC / 4)), r = rem / (TC / 4), c = (rem - r * (TC / 4)) * 4;
            float f[4];
            bytes4_to_float(b_raw[k], f);
            *reinterpret_cast<float4*>(&b_sh[buf][pp][r][c]) = make_float4(f[0], f[1], f[2], f[3]);
        }
        if (tid < PC) w_sh[buf][tid] = w_raw;
    };

    float z[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) z[i][j] = 0.0f;

    fetch(0);
    stage(0);
    __syncthreads();
    int buf = 0;
    for (int p0 = 0; p0 < pairs; p0 += PC, buf ^= 1) {
        const bool more = p0 + PC < pairs;
        if (more) fetch(p0 + PC);
        const int cnt = min(PC, pairs - p0);
#pragma unroll 4
        for (int pp = 0; pp < cnt; ++pp) {
            const float w = w_sh[buf][pp];
            float e[4][4];
#pragma unroll
            for (int r = 0; r < RANK; ++r) {
                const float4 a4 = *reinterpret_cast<const float4*>(&a_sh[buf][pp][r][ty * 4]);
                const float4 b4 = *reinterpret_cast<const float4*>(&b_sh[buf][pp][r][tx * 4]);
                const float av[4] = {a4.x, a4.y, a4.z, a4.w}, bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) e[i][j] = r == 0 ? __fmul_rn(av[i], bv[j]) : fmaf(av[i], bv[j], e[i][j]);  // exact: small integers
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) z[i][j] = fmaf(w, e[i][j], z[i][j]);
        }
        if (more) stage(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = row_base + ty * 4 + i;
        if (row >= row_end) continue;
        float* dst = d.Z + static_cast<size_t>(row) * d.cols + col_base + tx * 4;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (col_base + tx * 4 + j < d.cols) dst[j] = __fmul_rn(cscale, z[i][j]);
    }
}

// Sum of squares, stage 1: the squares of 256 consecutive elements are added in the order of the reference's shared-memory tree
// (strides 128, 64, .. 1). One warp per 256 elements: lane l holds elements l, l + 32, .. so that the strides down to 32 are
// register additions and the rest shuffles; no barriers, eight loads in flight per lane.
__device__ __forceinline__ float sumsq_256(const float* Z, int first, int n) {
    const int lane = threadIdx.x & 31;
    float e[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int i = first + lane + 32 * j;
        const float z = i < n ? Z[i] : 0.0f;
        e[j] = __fmul_rn(z, z);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] += e[j + 4];
    e[0] += e[2];
    e[1] += e[3];
    e[0] += e[1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e[0] += __shfl_down_sync(0xffffffffu, e[0], o);
    return e[0];  // lane 0
}
__global__ void __launch_bounds__(256) sumsq_blocks_kernel(const float* __restrict__ Z, int n, float* __restrict__ partial) {
    pdl_wait();
    after(Z);
    const int block = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (block * 256ll >= n) return;
    const float t = sumsq_256(Z, block * 256, n);
    if ((threadIdx.x & 31) == 0) partial[block] = t;
}
// stage 2: the block partials in double, in a fixed order (256 strided chains, then a tree). Result in thread 0.
__device__ __forceinline__ double sumsq_total(const float* partial, int nblocks) {
    __shared__ double warp_sum[8];
    double t = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += 256) t += static_cast<double>(partial[b]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < 8; ++w) t += warp_sum[w];
    return t;
}
__global__ void __launch_bounds__(256) sumsq_final_kernel(const float* __restrict__ partial, int nblocks, float* sumsq) {
    pdl_wait();
    after(partial);
    const double tot = sumsq_total(partial, nblocks);
    if (threadIdx.x == 0) sumsq[0] += static_cast<float>(tot);
}

__global__ void inv_rms_kernel(const float* __restrict__ sumsq, float* __restrict__ rms_ema, int use_adaptive, float beta, float eps,
                               int n, float* __restrict__ inv_rms_out) {
    pdl_wait();
    after(sumsq);
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    float inv = 1.0f;
    if (use_adaptive) {
        const float ms = __fdiv_rn(sumsq[0], static_cast<float>(n));
        float ema = rms_ema[0];
        if (ema == 0.0f) ema = ms;
        ema = fmaf(beta, ema, __fmul_rn(1.0f - beta, ms));
        rms_ema[0] = ema;
        inv = __fdiv_rn(1.0f, __fsqrt_rn(ema + eps));
    }
    inv_rms_out[0] = inv;
}

__global__ void update_shadow_kernel(int8_t* __restrict__ w, float* __restrict__ shadow, const float* __restrict__ Z, int n,
                                     const float* __restrict__ inv_rms_dev, float inv_rms_host, float lr, float thresh) {
    pdl_wait();
    after(Z, inv_rms_dev);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float inv = inv_rms_dev != nullptr ? inv_rms_dev[0] : inv_rms_host;
    const float g = __fmul_rn(inv, Z[i]);
    if (fabsf(g) < thresh) return;
    const float s = fmaf(lr, g, shadow[i]);
    shadow[i] = s;
    w[i] = static_cast<int8_t>(clip_ternary(__float2int_rn(s)));
}

__global__ void update_vector_kernel(float* __restrict__ v, const float* __restrict__ Z, int n, const float* __restrict__ inv_rms,
                                     float lr, float thresh) {
    pdl_wait();
    after(Z, inv_rms);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = __fmul_rn(inv_rms[0], Z[i]);
    if (fabsf(g) < thresh) return;
    v[i] = fmaf(lr, g, v[i]);
}

__global__ void add_scaled_kernel(float* __restrict__ out, const float* __restrict__ noise, int n, float scale) {
    pdl_wait();
    after(noise);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = fmaf(scale, noise[i], out[i]);
}

// Fitness shaping on the device, bit for bit the host function bnf4_shape_pair_weights (api.cu): f_p = -(loss+ - loss-), then sign,
// z-score or centered rank followed by the z-score with clipping. Ranks come from counting (ties by index, as the stable sort
// orders them); mean and variance are sums in index order, one thread each way, because that is the order the host adds in (1024
// pairs: about 5 us, against a stream synchronisation, two copies and an idle GPU between evaluation and update).
constexpr int kShapeMaxPairs = 4096;
__global__ void __launch_bounds__(1024) shape_fitness_kernel(const float* __restrict__ losses, int n, int mode, float clip, float* __restrict__ out) {
    pdl_wait();
    after(losses);
    __shared__ float f[kShapeMaxPairs], r[kShapeMaxPairs];
    __shared__ float mean_s, std_s;
    for (int i = threadIdx.x; i < n; i += 1024) f[i] = -__fsub_rn(losses[2 * i], losses[2 * i + 1]);
    __syncthreads();
    if (mode == BNF4_FITNESS_SIGN) {
        for (int i = threadIdx.x; i < n; i += 1024) out[i] = f[i] > 0.0f ? 1.0f : (f[i] < 0.0f ? -1.0f : 0.0f);
        return;
    }
    for (int i = threadIdx.x; i < n; i += 1024) {
        float v = f[i];
        if (mode == BNF4_FITNESS_CENTERED_RANK) {
            int rank = 0;
            for (int j = 0; j < n; ++j) rank += (f[j] < v || (j < i && !(v < f[j]))) ? 1 : 0;
            v = n == 1 ? 0.0f : __fsub_rn(__fdiv_rn(static_cast<float>(rank), static_cast<float>(n - 1)), 0.5f);
        }
        r[i] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float mean = 0.0f;
#pragma unroll 16
        for (int i = 0; i < n; ++i) mean = __fadd_rn(mean, r[i]);
        mean = __fdiv_rn(mean, static_cast<float>(n));
        mean_s = mean;
    }
    __syncthreads();
    const float mean = mean_s;
    for (int i = threadIdx.x; i < n; i += 1024) {
        const float d = __fsub_rn(r[i], mean);
        r[i] = d;
        f[i] = __fmul_rn(d, d);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float var = 0.0f;
#pragma unroll 16
        for (int i = 0; i < n; ++i) var = __fadd_rn(var, f[i]);
        std_s = __fadd_rn(__fsqrt_rn(__fdiv_rn(var, static_cast<float>(n))), 1e-6f);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += 1024) {
        float d = __fdiv_rn(r[i], std_s);
        if (d > clip) d = clip;
        if (d < -clip) d = -clip;
        out[i] = d;
    }
}

// ---- the apply phase of the ES update for a table of tensors: three launches for all of them ----------------------------------
// Same arithmetic and summation order as sumsq_blocks / sumsq_final / inv_rms / update_shadow / update_vector above, so the bits are
// those of the per-tensor calls. The tensor of a block is found by binary search over the running block counts.
template <bool UPDATE_BLOCKS>
__device__ __forceinline__ int find_tensor(const UpdApplyDesc* __restrict__ d, int ndesc, int block) {
    int lo = 0, hi = ndesc - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((UPDATE_BLOCKS ? d[mid].ublock0 : d[mid].block0) <= block) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__global__ void __launch_bounds__(256) sumsq_blocks_batched_kernel(const UpdApplyDesc* __restrict__ d, int ndesc, int total_blocks,
                                                                   const float* __restrict__ z_all, float* __restrict__ partial) {
    pdl_wait();
    after(z_all);
    const int block = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (block >= total_blocks) return;
    const UpdApplyDesc& x = d[find_tensor<false>(d, ndesc, block)];
    const float t = sumsq_256(z_all + x.zoff, (block - x.block0) * 256, x.n);
    if ((threadIdx.x & 31) == 0) partial[block] = t;
}
// one CTA per tensor; its thread 0 turns the sum into inv_rms (and advances the tensor's RMS-EMA)
__global__ void __launch_bounds__(256) sumsq_final_inv_rms_batched_kernel(const UpdApplyDesc* __restrict__ d, const float* __restrict__ partial, int use_adaptive,
                                                                          float beta, float eps, float* __restrict__ inv_rms_out) {
    pdl_wait();
    after(partial);
    const UpdApplyDesc& x = d[blockIdx.x];
    const double tot = sumsq_total(partial + x.block0, (x.n + 255) / 256);
    if (threadIdx.x != 0) return;
    float inv = 1.0f;
    if (use_adaptive) {
        const float ms = __fdiv_rn(static_cast<float>(tot), static_cast<float>(x.n));
        float ema = x.ema[0];
        if (ema == 0.0f) ema = ms;
        ema = fmaf(beta, ema, __fmul_rn(1.0f - beta, ms));
        x.ema[0] = ema;
        inv = __fdiv_rn(1.0f, __fsqrt_rn(ema + eps));
    }
    inv_rms_out[blockIdx.x] = inv;
}
// Gated update of four consecutive elements per thread (16-byte accesses, a warp covers 512 contiguous bytes of Z and shadow) and,
// in the same pass, the NVFP4 copy of the new weights: the four threads of a 16-element scale block agree on its maximum with two
// shuffles. Memory bound: 14 bytes per weight read and written plus 0.56 of NVFP4, against a second pass over the weights by one
// quantiser launch per matrix. UPDATE false: the NVFP4 copies of the present weights only.
template <bool UPDATE>
__global__ void __launch_bounds__(256) update_batched_kernel(const UpdApplyDesc* __restrict__ d, int ndesc, const float* __restrict__ z_all,
                                                             const float* __restrict__ inv_rms, float lr, float thresh, const uint2* __restrict__ tab) {
    pdl_wait();
    after(z_all, inv_rms);
    const int ti = find_tensor<true>(d, ndesc, static_cast<int>(blockIdx.x));
    const UpdApplyDesc& x = d[ti];
    const int i0 = (static_cast<int>(blockIdx.x) - x.ublock0) * 1024 + static_cast<int>(threadIdx.x) * 4;
    const int n = x.n;
    int8_t* w = x.w;
    uint32_t wq = 0;  // the four weights as bytes
    const bool whole = i0 + 4 <= n;
    if constexpr (UPDATE) {
        const float* Z = z_all + x.zoff;
        float* target = x.target;
        const float inv = inv_rms[ti];
        if (whole && ((reinterpret_cast<uintptr_t>(Z) | reinterpret_cast<uintptr_t>(target)) & 15) == 0) {
            const float4 z4 = *reinterpret_cast<const float4*>(Z + i0);
            float4 s4 = *reinterpret_cast<const float4*>(target + i0);
            uint32_t old = w != nullptr ? *reinterpret_cast<const uint32_t*>(w + i0) : 0u;
            const float zz[4] = {z4.x, z4.y, z4.z, z4.w};
            float ss[4] = {s4.x, s4.y, s4.z, s4.w};
            bool any = false;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float g = __fmul_rn(inv, zz[e]);
                if (!(fabsf(g) < thresh)) {
                    any = true;
                    ss[e] = fmaf(lr, g, ss[e]);
                    old = (old & ~(0xffu << (8 * e))) | (static_cast<uint32_t>(clip_ternary(__float2int_rn(ss[e])) & 0xff) << (8 * e));
                }
            }
            if (any) {
                *reinterpret_cast<float4*>(target + i0) = make_float4(ss[0], ss[1], ss[2], ss[3]);
                if (w != nullptr) *reinterpret_cast<uint32_t*>(w + i0) = old;
            }
            wq = old;
        } else {
            for (int i = i0; i < min(n, i0 + 4); ++i) {
                const float g = __fmul_rn(inv, Z[i]);
                if (!(fabsf(g) < thresh)) {
                    const float s = fmaf(lr, g, target[i]);
                    target[i] = s;
                    if (w != nullptr) w[i] = static_cast<int8_t>(clip_ternary(__float2int_rn(s)));
                }
                if (w != nullptr) wq |= static_cast<uint32_t>(static_cast<uint8_t>(w[i])) << (8 * (i - i0));
            }
        }
    } else {
        if (w != nullptr && whole) wq = *reinterpret_cast<const uint32_t*>(w + i0);
    }
    if (x.codes == nullptr) return;  // (uniform in the CTA; matrices with a copy have n a multiple of 16)
    float f[4];
    bytes4_to_float(wq, f);
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = fmaxf(f[e], -127.0f);  // -128 is treated as -127, as by the row quantisers
    float am = fmaxf(fmaxf(fabsf(f[0]), fabsf(f[1])), fmaxf(fabsf(f[2]), fabsf(f[3])));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 2));
    if (i0 >= n) return;
    const uint2 ent = __ldg(tab + x.scaled * 128 + static_cast<int>(am));
    const float n8[8] = {f[0], f[1], f[2], f[3], 0.0f, 0.0f, 0.0f, 0.0f};
    const uint32_t codes = e2m1x8_int(n8, __uint_as_float(ent.x));
    const int row = i0 / x.cols, col = i0 - row * x.cols;
    *reinterpret_cast<uint16_t*>(x.codes + (static_cast<size_t>(x.row0 + row) * x.cols + col) / 2) = static_cast<uint16_t>(codes);
    if ((col & 15) == 0) x.sf[sf_offset(x.row0 + row, col >> 4, sf_k_atoms(x.cols))] = static_cast<uint8_t>(ent.y);
}

// library-owned scratch for the block partials of sum(Z^2), one per device
struct Scratch {
    float* ptr = nullptr;
    size_t floats = 0;
};
std::mutex g_scratch_mu;
Scratch g_scratch[64];

int get_scratch(size_t floats, float** out) {
    int dev = 0;
    int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (dev < 0 || dev >= 64) return set_error(BNF4_ERR_INVALID, "device index %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    Scratch& s = g_scratch[dev];
    if (s.floats < floats) {
        // stream-ordered users of the old buffer may still be running: synchronise before freeing it
        if (s.ptr != nullptr) {
            rc = check_cuda(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
            if (rc) return rc;
            cudaFree(s.ptr);
            s.ptr = nullptr;
            s.floats = 0;
        }
        const size_t want = floats < 65536 ? 65536 : floats;
        rc = check_cuda(cudaMalloc(&s.ptr, want * sizeof(float)), "cudaMalloc(sumsq scratch)");
        if (rc) return rc;
        s.floats = want;
    }
    *out = s.ptr;
    return BNF4_OK;
}

}  // namespace

int cross_entropy_launch(const float* logits, int ld, const float* bias, const int8_t* bias_noise, float sigma, const uint8_t* targets, int vocab, int members,
                         int rows_per_member, float* partial, unsigned* counters, float* loss_mean, cudaStream_t st) {
    // few members (a validation pass has one): more blocks per member as long as the SMs are not filled and a warp keeps four rows. Same bits. One member of
    // 4096 rows, end of its whole pass: 63.5 us with at most four, 61.6 with eight; of 16384 rows 164 and 150.
    int split = 1;
    while (counters != nullptr && split < 8 && members * kCeChunks * split < 2 * 148 && rows_per_member >= 2 * split * 512) split *= 2;
    const dim3 grid(kCeChunks * split, members);
    const bool early = static_cast<long long>(members) * rows_per_member * vocab <= kPdlStreamElems;
    const bool vec = (vocab % 4) == 0 && (ld % 4) == 0 && ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(bias)) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(bias_noise) & 3) == 0;
    auto run = [&](auto kernel) { launch_pdl_if(early, kernel, grid, 256, 0, st, logits, ld, bias, bias_noise, sigma, targets, vocab, rows_per_member, partial, counters, loss_mean); };
    auto pick = [&](auto shared) {
        constexpr bool SH = decltype(shared)::value;
        if (vec && vocab <= 128) run(ce_population_vec_kernel<1, 4, SH>);
        else if (vec && vocab <= 256) run(ce_population_vec_kernel<2, 4, SH>);
        else if (vec && vocab <= 512) run(ce_population_vec_kernel<4, 2, SH>);
        else if (vec) run(ce_population_vec_kernel<8, 1, SH>);
        else run(ce_population_kernel<SH>);
    };
    if (split > 1) pick(std::true_type());
    else pick(std::false_type());
    return check_launch("ce_population_kernel");
}

bool shape_fitness_applies(int pairs, int mode) { return pairs <= kShapeMaxPairs && mode >= BNF4_FITNESS_SIGN && mode <= BNF4_FITNESS_CENTERED_RANK; }
int shape_fitness_launch(const float* losses, int pairs, int mode, float clip, float* weights, cudaStream_t st) {
    launch_pdl(shape_fitness_kernel, 1, 1024, 0, st, losses, pairs, mode, clip, weights);
    return check_launch("shape_fitness_kernel");
}

namespace {
// 524288 elements x 1024 pairs: 2.87 ms with the generic hash (branches on the noise kind, a loop over the draws), 2.22 ms with the
// specialised one; both are bound by the integer pipes.
int z_dense_single(const float* pair_weights, const uint64_t* pair_seeds, uint64_t salt, int pairs, int n, int use_clt, int clt_k, float* Z, cudaStream_t st) {
    const bool early = static_cast<long long>(n) * pairs <= (1ll << 22);
    const dim3 grid((n + 255) / 256);
    if (use_clt != 0 && clt_k == 4) launch_pdl_if(early, z_dense_kernel<true>, grid, 256, 0, st, pair_weights, pair_seeds, salt, pairs, n, use_clt, clt_k, Z);
    else launch_pdl_if(early, z_dense_kernel<false>, grid, 256, 0, st, pair_weights, pair_seeds, salt, pairs, n, use_clt, clt_k, Z);
    return check_launch("z_dense_kernel");
}
}  // namespace

int z_dense_table_launch(const float* pair_weights, const uint64_t* pair_seeds, const ZDenseDesc* d_descs, const ZDenseDesc* h_descs, int ndesc, int pairs,
                         int use_clt, int clt_k, int shard, int nshards, float* z_all, cudaStream_t st) {
    long long blocks = 0, elems = 0;
    for (int i = 0; i < ndesc; ++i) {
        int i0 = 0, cnt = 0;
        z_dense_range(h_descs[i], shard, nshards, i0, cnt);
        blocks += (cnt + 255) / 256;
        elems += cnt;
    }
    if (blocks <= 0) return BNF4_OK;
    const bool early = elems * pairs <= (1ll << 22);
    const dim3 grid(static_cast<unsigned>(blocks));
    if (use_clt != 0 && clt_k == 4)
        launch_pdl_if(early, z_dense_table_kernel<true>, grid, 256, 0, st, pair_weights, pair_seeds, d_descs, ndesc, pairs, use_clt, clt_k, shard, nshards, z_all);
    else
        launch_pdl_if(early, z_dense_table_kernel<false>, grid, 256, 0, st, pair_weights, pair_seeds, d_descs, ndesc, pairs, use_clt, clt_k, shard, nshards, z_all);
    return check_launch("z_dense_table_kernel");
}

void update_quant_table(float row_scale, float up, uint2 (&tab)[256]) {
    for (int scaled = 0; scaled < 2; ++scaled)
        for (int amax = 0; amax < 128; ++amax) {  // the arithmetic of quant_block16, IEEE on host and device alike
            float scale = amax > 0 ? static_cast<float>(amax) / 6.0f : 1.0f;
            if (scaled) scale *= row_scale;
            uint32_t sq = ue4m3_encode_host(scale);
            float sf = ue4m3_decode(sq);
            if (sf == 0.0f) { sq = 0x38u; sf = 1.0f; }
            const float rcp = 1.0f / sf;
            uint2 e;
            memcpy(&e.x, &rcp, 4);
            e.y = up == 1.0f ? sq : ue4m3_encode_host(sf * up);
            tab[scaled * 128 + amax] = e;
        }
}

// Apply phase for a table of tensors; partial holds one float per 256-element block, inv_rms one per tensor.
int update_apply_batched(const UpdApplyDesc* d_descs, int ndesc, int total_blocks, int total_ublocks, const float* z_all, const uint2* tab, float* partial,
                         float* inv_rms, int use_adaptive, float beta, float eps, float lr, float thresh, cudaStream_t st) {
    if (ndesc <= 0 || total_blocks <= 0) return BNF4_OK;
    const bool early = total_blocks * 256ll <= kPdlStreamElems;
    launch_pdl_if(early, sumsq_blocks_batched_kernel, (total_blocks + 7) / 8, 256, 0, st, d_descs, ndesc, total_blocks, z_all, partial);
    int rc = check_launch("sumsq_blocks_batched_kernel");
    if (rc) return rc;
    launch_pdl(sumsq_final_inv_rms_batched_kernel, ndesc, 256, 0, st, d_descs, partial, use_adaptive, beta, eps, inv_rms);
    rc = check_launch("sumsq_final_inv_rms_batched_kernel");
    if (rc) return rc;
    launch_pdl_if(early, update_batched_kernel<true>, total_ublocks, 256, 0, st, d_descs, ndesc, z_all, inv_rms, lr, thresh, tab);
    return check_launch("update_batched_kernel");
}
int requantize_batched(const UpdApplyDesc* d_descs, int ndesc, int total_ublocks, const uint2* tab, cudaStream_t st) {
    launch_pdl(update_batched_kernel<false>, total_ublocks, 256, 0, st, d_descs, ndesc, nullptr, nullptr, 0.0f, 0.0f, tab);
    return check_launch("update_batched_kernel");
}

// d_descs: the table in device memory (nullptr with ndesc == 0: the single matrix h_descs[0], passed by value).
// h_descs: the same table in host memory, for the grid size.
int z_lowrank_launch(const float* pair_weights, const ZLowrankDesc* d_descs, const ZLowrankDesc* h_descs, int ndesc, int pairs, int rank,
                     float cscale, int shard, int nshards, ZTables tables, const ZDenseDesc* h_tables, cudaStream_t st) {
    if (rank < 1 || rank > 4) return set_error(BNF4_ERR_INVALID, "compute_z_lowrank: rank=%d outside [1,4]", rank);
    if (nshards < 1 || shard < 0 || shard >= nshards) return set_error(BNF4_ERR_INVALID, "compute_z_lowrank: shard %d of %d", shard, nshards);
    if (pairs <= 0) return set_error(BNF4_ERR_INVALID, "compute_z_lowrank: pairs=%d", pairs);
    long long tiles = 0;
    for (int i = 0; i < std::max(ndesc, 1); ++i) {
        int nr = h_descs[i].rows;
        if (ndesc > 0 && nshards > 1 && nr >= nshards && (nr % nshards) == 0) nr /= nshards;
        tiles += static_cast<long long>((nr + kZTileRows - 1) / kZTileRows) * ((h_descs[i].cols + kZTileCols - 1) / kZTileCols);
    }
    tables.blocks = 0;
    for (int i = 0; i < tables.ndesc; ++i) {
        int i0 = 0, cnt = 0;
        z_dense_range(h_tables[i], shard, nshards, i0, cnt);
        tables.blocks += (cnt + kZThreads - 1) / kZThreads;
    }
    tiles += tables.blocks;
    if (tiles <= 0) return BNF4_OK;
    if (tiles > 0x7fffffffLL) return set_error(BNF4_ERR_INVALID, "compute_z_lowrank: too many tiles");
    const unsigned grid = static_cast<unsigned>(tiles);
    const ZLowrankDesc single = h_descs[0];
    switch (rank) {
        case 1: launch_pdl_if(grid <= 2048, z_lowrank_tiles_kernel<1>, grid, kZThreads, 0, st, pair_weights, d_descs, ndesc, single, pairs, cscale, shard, nshards, tables); break;
        case 2: launch_pdl_if(grid <= 2048, z_lowrank_tiles_kernel<2>, grid, kZThreads, 0, st, pair_weights, d_descs, ndesc, single, pairs, cscale, shard, nshards, tables); break;
        case 3: launch_pdl_if(grid <= 2048, z_lowrank_tiles_kernel<3>, grid, kZThreads, 0, st, pair_weights, d_descs, ndesc, single, pairs, cscale, shard, nshards, tables); break;
        default: launch_pdl_if(grid <= 2048, z_lowrank_tiles_kernel<4>, grid, kZThreads, 0, st, pair_weights, d_descs, ndesc, single, pairs, cscale, shard, nshards, tables); break;
    }
    return check_launch("z_lowrank_tiles_kernel");
}

namespace {

int sumsq_into(const float* Z, int n, float* sumsq, cudaStream_t st) {
    const int nblocks = (n + 255) / 256;
    float* partial = nullptr;
    int rc = get_scratch(static_cast<size_t>(nblocks), &partial);
    if (rc) return rc;
    launch_pdl(sumsq_blocks_kernel, (nblocks + 7) / 8, 256, 0, st, Z, n, partial);
    rc = check_launch("sumsq_blocks_kernel");
    if (rc) return rc;
    launch_pdl(sumsq_final_kernel, 1, 256, 0, st, partial, nblocks, sumsq);
    return check_launch("sumsq_final_kernel");
}

}  // namespace

int sumsq_with_scratch(const float* Z, int n, float* partial, float* sumsq, cudaStream_t st) {
    const int nblocks = (n + 255) / 256;
    launch_pdl(sumsq_blocks_kernel, (nblocks + 7) / 8, 256, 0, st, Z, n, partial);
    int rc = check_launch("sumsq_blocks_kernel");
    if (rc) return rc;
    launch_pdl(sumsq_final_kernel, 1, 256, 0, st, partial, nblocks, sumsq);
    return check_launch("sumsq_final_kernel");
}

}  // namespace bnf4

using namespace bnf4;
static inline cudaStream_t S(void* s) { return static_cast<cudaStream_t>(s); }

extern "C" {

int bnf4_cross_entropy_loss(const float* logits, const float* bias, const float* bias_noise, float bias_noise_scale,
                            const uint8_t* targets_t, int token_stride, int vocab, int batch, float* loss_accum, void* stream) {
    if (batch <= 0) return BNF4_OK;
    if (!logits || !targets_t || !loss_accum) return set_error(BNF4_ERR_INVALID, "cross_entropy_loss: null pointer");
    if (vocab <= 0 || vocab > 32 * kCeMaxPerLane) return set_error(BNF4_ERR_INVALID, "cross_entropy_loss: vocab=%d outside [1,%d]", vocab, 32 * kCeMaxPerLane);
    launch_pdl(ce_step_kernel, 1, 1024, 0, S(stream), logits, bias, bias_noise, bias_noise_scale, targets_t, token_stride, vocab, batch, loss_accum);
    return check_launch("ce_step_kernel");
}

int bnf4_cross_entropy_population(const float* logits, int ld, const float* bias, const int8_t* bias_noise, float sigma,
                                  const uint8_t* targets, int vocab, int members, int rows_per_member, float* partial,
                                  float* loss_mean, void* stream) {
    if (members <= 0 || rows_per_member <= 0) return BNF4_OK;
    if (!logits || !targets || !partial || !loss_mean) return set_error(BNF4_ERR_INVALID, "cross_entropy_population: null pointer");
    if (vocab <= 0 || vocab > 32 * kCeMaxPerLane) return set_error(BNF4_ERR_INVALID, "cross_entropy_population: vocab=%d", vocab);
    if (members > 65535) return set_error(BNF4_ERR_INVALID, "cross_entropy_population: at most 65535 members per call");
    int rc = cross_entropy_launch(logits, ld, bias, bias_noise, sigma, targets, vocab, members, rows_per_member, partial, nullptr, loss_mean, S(stream));
    if (rc) return rc;
    launch_pdl(ce_finalize_kernel, (members + 127) / 128, 128, 0, S(stream), partial, members, rows_per_member, loss_mean);
    return check_launch("ce_finalize_kernel");
}

int bnf4_fill_ternary_noise(int8_t* out, size_t n, uint64_t seed, int use_clt, int clt_k, void* stream) {
    if (n == 0) return BNF4_OK;
    if (!out) return set_error(BNF4_ERR_INVALID, "fill_ternary_noise: null pointer");
    launch_pdl(fill_noise_kernel, static_cast<unsigned>((n + 255) / 256), 256, 0, S(stream), out, n, seed, use_clt, clt_k);
    return check_launch("fill_noise_kernel");
}

int bnf4_fill_ternary_noise_batched(const bnf4_noise_desc* descs, int num_desc, int max_blocks, int use_clt, int clt_k, void* stream) {
    if (num_desc <= 0 || max_blocks <= 0) return BNF4_OK;
    if (!descs) return set_error(BNF4_ERR_INVALID, "fill_ternary_noise_batched: null pointer");
    launch_pdl(fill_noise_batched_kernel, dim3(max_blocks, num_desc), 256, 0, S(stream), descs, num_desc, use_clt, clt_k);
    return check_launch("fill_noise_batched_kernel");
}

int bnf4_fill_float_noise(float* out, int n, uint64_t seed, int use_clt, int clt_k, void* stream) {
    if (n <= 0) return BNF4_OK;
    launch_pdl(fill_float_noise_kernel, (n + 255) / 256, 256, 0, S(stream), out, n, seed, use_clt, clt_k);
    return check_launch("fill_float_noise_kernel");
}

int bnf4_init_shadow_from_weights(const int8_t* w, float* shadow, int n, void* stream) {
    if (n <= 0) return BNF4_OK;
    launch_pdl(init_shadow_kernel, (n + 255) / 256, 256, 0, S(stream), w, shadow, n);
    return check_launch("init_shadow_kernel");
}

int bnf4_fill_pair_seeds(uint64_t base_seed, uint64_t epoch, int pairs, uint64_t* out, void* stream) {
    if (pairs <= 0) return BNF4_OK;
    launch_pdl(pair_seeds_kernel, (pairs + 255) / 256, 256, 0, S(stream), base_seed, epoch, pairs, out);
    return check_launch("pair_seeds_kernel");
}

int bnf4_compute_z_sumsq(const float* pair_weights, const uint64_t* pair_seeds, uint64_t salt, int pairs, int n, int use_clt,
                         int clt_k, float* Z, float* sumsq, void* stream) {
    if (n <= 0) return BNF4_OK;
    if (!pair_weights || !pair_seeds || !Z || !sumsq) return set_error(BNF4_ERR_INVALID, "compute_z_sumsq: null pointer");
    const int rc = z_dense_single(pair_weights, pair_seeds, salt, pairs, n, use_clt, clt_k, Z, S(stream));
    if (rc) return rc;
    return sumsq_into(Z, n, sumsq, S(stream));
}

int bnf4_compute_z_lowrank(const float* pair_weights, const int8_t* A, long long A_pair_stride, const int8_t* B,
                           long long B_pair_stride, int pairs, int rows, int cols, int rank, float cscale, float* Z, void* stream) {
    if (rows <= 0 || cols <= 0) return BNF4_OK;
    if (!pair_weights || !A || !B || !Z) return set_error(BNF4_ERR_INVALID, "compute_z_lowrank: null pointer");
    const ZLowrankDesc d = {A, A_pair_stride, B, B_pair_stride, Z, rows, cols};
    return z_lowrank_launch(pair_weights, nullptr, &d, 0, pairs, rank, cscale, 0, 1, ZTables{}, nullptr, S(stream));
}

int bnf4_sumsq(const float* Z, int n, float* sumsq, void* stream) {
    if (n <= 0) return BNF4_OK;
    if (!Z || !sumsq) return set_error(BNF4_ERR_INVALID, "sumsq: null pointer");
    return sumsq_into(Z, n, sumsq, S(stream));
}

int bnf4_compute_z_sumsq_lowrank(const float* pair_weights, const int8_t* A, long long A_pair_stride, const int8_t* B,
                                 long long B_pair_stride, int pairs, int rows, int cols, int rank, float cscale, float* Z,
                                 float* sumsq, void* stream) {
    if (rows <= 0 || cols <= 0) return BNF4_OK;
    if (!sumsq) return set_error(BNF4_ERR_INVALID, "compute_z_sumsq_lowrank: null pointer");
    const int rc = bnf4_compute_z_lowrank(pair_weights, A, A_pair_stride, B, B_pair_stride, pairs, rows, cols, rank, cscale, Z, stream);
    if (rc) return rc;
    return sumsq_into(Z, rows * cols, sumsq, S(stream));
}

int bnf4_update_inv_rms(const float* sumsq, float* rms_ema, int use_adaptive, float adaptive_beta, float adaptive_eps, int n,
                        float* inv_rms, void* stream) {
    if (!sumsq || !rms_ema || !inv_rms) return set_error(BNF4_ERR_INVALID, "update_inv_rms: null pointer");
    launch_pdl(inv_rms_kernel, 1, 1, 0, S(stream), sumsq, rms_ema, use_adaptive, adaptive_beta, adaptive_eps, n, inv_rms);
    return check_launch("inv_rms_kernel");
}

int bnf4_update_shadow_ternary_device(int8_t* w, float* shadow, const float* Z, int n, const float* inv_rms, float lr,
                                      float thresh, void* stream) {
    if (n <= 0) return BNF4_OK;
    if (!inv_rms) return set_error(BNF4_ERR_INVALID, "update_shadow_ternary_device: null inv_rms");
    launch_pdl(update_shadow_kernel, (n + 255) / 256, 256, 0, S(stream), w, shadow, Z, n, inv_rms, 0.0f, lr, thresh);
    return check_launch("update_shadow_kernel");
}

int bnf4_update_shadow_ternary(int8_t* w, float* shadow, const float* Z, int n, float inv_rms, float lr, float thresh, void* stream) {
    if (n <= 0) return BNF4_OK;
    launch_pdl(update_shadow_kernel, (n + 255) / 256, 256, 0, S(stream), w, shadow, Z, n, nullptr, inv_rms, lr, thresh);
    return check_launch("update_shadow_kernel");
}

int bnf4_update_vector_device(float* v, const float* Z, int n, const float* inv_rms, float lr, float thresh, void* stream) {
    if (n <= 0) return BNF4_OK;
    launch_pdl(update_vector_kernel, (n + 255) / 256, 256, 0, S(stream), v, Z, n, inv_rms, lr, thresh);
    return check_launch("update_vector_kernel");
}

int bnf4_add_scaled(float* out, const float* noise, int n, float scale, void* stream) {
    if (n <= 0) return BNF4_OK;
    launch_pdl(add_scaled_kernel, (n + 255) / 256, 256, 0, S(stream), out, noise, n, scale);
    return check_launch("add_scaled_kernel");
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------
// bnf4_compute_z_sumsq_static: the dense Z / sum-of-squares step with no allocation of any kind.
//
// bnf4_compute_z_sumsq keeps its block partials in a buffer the library obtains from cudaMalloc the first time
// it is needed on a device and replaces by a larger one when a longer vector arrives. Some hosts cannot accept
// that: a trainer whose own allocator has already reserved the whole of HBM (a library cudaMalloc then fails
// although the job has memory to spare), a serving loop in which the implicit device-wide synchronisation of
// cudaMalloc / cudaFree stalls every other stream, or a process that must keep a fixed, auditable device
// footprint. For them the partials live in the array below, which is part of the loaded module image: it exists
// as soon as the library is loaded on a device and is never resized or released.
//
// Capacity: kStaticPartials block partials of 256 elements each, i.e. n <= 67,108,864 (an 8192 x 8192 matrix);
// longer vectors are refused with BNF4_ERR_INVALID and nothing is launched.
// ---------------------------------------------------------------------------------------------------
static constexpr int kStaticPartials = 262144;  // 1 MiB of device memory per device
static constexpr long long kStaticMaxN = 256LL * kStaticPartials;
static __device__ __align__(256) float g_static_partials[kStaticPartials];

namespace {
std::mutex g_static_mu;
float* g_static_ptr[64] = {};  // device address of g_static_partials, per device ordinal; filled on first use

// Resolves the device address of the array for the CURRENT device (each device holds its own copy of a
// __device__ variable). Host code never uses the array's name as an address: only the pointer obtained here
// is handed to kernels.
int static_partials(float** out) {
    int dev = 0;
    int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (dev < 0 || dev >= 64) return set_error(BNF4_ERR_INVALID, "device index %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (g_static_ptr[dev] == nullptr) {
        float* ptr = nullptr;
        rc = check_cuda(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_partials), "cudaGetSymbolAddress(static partials)");
        if (rc) return rc;
        if (ptr == nullptr) return set_error(BNF4_ERR_CUDA, "cudaGetSymbolAddress returned a null address");
        g_static_ptr[dev] = ptr;
    }
    *out = g_static_ptr[dev];
    return BNF4_OK;
}
}  // namespace

extern "C" int bnf4_compute_z_sumsq_static(const float* pair_weights, const uint64_t* pair_seeds, uint64_t salt, int pairs, int n,
                                           int use_clt, int clt_k, float* Z, float* sumsq, void* stream) {
    if (n <= 0) return BNF4_OK;
    if (!pair_weights || !pair_seeds || !Z || !sumsq) return set_error(BNF4_ERR_INVALID, "compute_z_sumsq_static: null pointer");
    if (static_cast<long long>(n) > kStaticMaxN)
        return set_error(BNF4_ERR_INVALID, "compute_z_sumsq_static: n=%d exceeds the built-in scratch capacity of %lld elements; "
                         "use bnf4_compute_z_sumsq or split the vector", n, kStaticMaxN);
    float* partial = nullptr;
    int rc = static_partials(&partial);
    if (rc) return rc;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    rc = z_dense_single(pair_weights, pair_seeds, salt, pairs, n, use_clt, clt_k, Z, st);
    if (rc) return rc;
    // Every partial the final kernel reads (indices 0 .. ceil(n/256)-1) is written by the block kernel of this same
    // call first, so stale contents left by an earlier call are never observed and nothing needs clearing.
    return sumsq_with_scratch(Z, n, partial, sumsq, st);
}
