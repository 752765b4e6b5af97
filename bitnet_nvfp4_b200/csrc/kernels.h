// Internal launcher interface between the translation units of the library (not installed).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "bnf4.h"

namespace bnf4 {

// ---------------------------------------------------------------------------------------------
// Row quantisers (rowquant.cu). Parameter block = the public bnf4_rowquant_desc.
// ---------------------------------------------------------------------------------------------
enum RowFrontEnd : int {
    FE_INT8 = BNF4_FE_INT8,                          // int8 rows in
    FE_WQKV = BNF4_FE_WQKV,                          // stacked [Wq;Wk;Wv;wbeta] rows, per-group scale folded into the block scale
    FE_EMBED_DENSE = BNF4_FE_EMBED_DENSE,            // emb[tok] + ns * noise[tok]
    FE_EMBED_LOWRANK = BNF4_FE_EMBED_LOWRANK,        // emb[tok] + ns*c_r * sum_r A[tok,r] B[j,r]
    FE_POS_GELU = BNF4_FE_POS_GELU,                  // gelu(in + pos) * act_scale
    FE_POS_GELU_ABSMEAN = BNF4_FE_POS_GELU_ABSMEAN,  // the above, kept as the residual stream, then abs-mean normalised
    FE_ACT = BNF4_FE_ACT,                            // none / relu / tanh / gelu*act_scale
    FE_ABSMEAN = BNF4_FE_ABSMEAN,                    // abs-mean norm of int8 rows
    FE_ADD_ABSMEAN = BNF4_FE_ADD_ABSMEAN,            // x8 = clip8(x8 + rint(y*add_scale)); abs-mean norm
};

constexpr int kMaxTVec = 16;  // rank-r projections per row (4 stacked groups x rank 4)

struct RowQuantParams : bnf4_rowquant_desc {
    RowQuantParams(const bnf4_rowquant_desc& d) : bnf4_rowquant_desc(d) {}
    int32_t* zero_t = nullptr;  // FE_ADD_ABSMEAN: clears [rows][zero_n] words, the projections the GEMM after next accumulates with atomics
    int zero_n = 0;
    int pad_sf = 0;              // also clears the padding of the scale array (rows to 128, columns to 64)
    int wide_ok = 0;  // set by the dispatch: the fp32 (or fp16) rows and the position table can be read 32 bytes at a time
    int batch = 1;    // set by the launch: rows a warp quantises before it takes their projections together
};
int rowquant_dispatch(int front_end, RowQuantParams p, cudaStream_t stream);

// ---------------------------------------------------------------------------------------------
// Block-scaled FP4 GEMM on tcgen05 (gemm_tcgen05.cu). Parameter block = the public bnf4_gemm_desc.
// ---------------------------------------------------------------------------------------------
enum GemmEpilogue : int {
    EPI_F32 = BNF4_EPI_F32,            // fp32 D
    EPI_GELU_I8 = BNF4_EPI_GELU_I8,    // int8 D = clip8(rint(gelu(v) * act_scale))
    EPI_GELU_FP4 = BNF4_EPI_GELU_FP4,  // the above re-quantised to e2m1 codes + ue4m3 scales (+ int8 copy, + t of the next GEMM)
    EPI_ADD_I8 = BNF4_EPI_ADD_I8,      // int8 residual stream updated in place: clip8(resid + rint(v * add_scale))
    EPI_F16 = BNF4_EPI_F16,            // leading columns as IEEE halves, the rest fp32
};

struct GemmParams : bnf4_gemm_desc {
    GemmParams() : bnf4_gemm_desc{} {}
    GemmParams(const bnf4_gemm_desc& d) : bnf4_gemm_desc(d) {}
    // Second B operand, accumulated after the first one over the same A: D += alpha A B2_member^T. [members][b2_rows][K] codes and their scale
    // atoms, b2_rows a multiple of 128; a member's rows (rows_per_member) are a multiple of 128.
    const void* b2 = nullptr;
    const void* sfb2 = nullptr;
    int b2_rows = 0;
};
int gemm_nvfp4_launch(const GemmParams& p, cudaStream_t stream);
// Reads and clears the device-side error word of the GEMM kernels (0 = none). Synchronises the stream.
int gemm_nvfp4_device_error(cudaStream_t stream, int* out_code);
extern int g_gemm_allow_tma_store;

// EFLA recurrence (efla.cu). Parameter block = the public bnf4_efla_desc.
struct EflaParams : bnf4_efla_desc {
    EflaParams() : bnf4_efla_desc{} {}
    EflaParams(const bnf4_efla_desc& d) : bnf4_efla_desc(d) {}
    // member_bias: the bias of sequence s is that of member m = s / seqs_per_bias, *beta_base + (+-bias_sigma) * bias_noise[(m / 2) * bias_stride]
    // with the sign of the member's parity (the per-member perturbation of a scalar; bias_sigma 0: no noise is read)
    int member_bias = 0;
    const float* beta_base = nullptr;
    const int8_t* bias_noise = nullptr;
    int bias_stride = 0;
    float bias_sigma = 0.0f;
};
#ifdef __CUDACC__
__device__ __forceinline__ float efla_seq_bias(const EflaParams& p, unsigned seq) {
    if (p.member_bias) {  // (reference: src/train_efla_lm.cpp:2912-2917)
        const unsigned member = seq / static_cast<unsigned>(p.seqs_per_bias);
        const float nz = p.bias_sigma != 0.0f ? static_cast<float>(p.bias_noise[static_cast<size_t>(member >> 1) * p.bias_stride]) : 0.0f;
        return fmaf((member & 1u) ? -p.bias_sigma : p.bias_sigma, nz, *p.beta_base);
    }
    return p.beta_bias_seq != nullptr ? p.beta_bias_seq[seq / static_cast<unsigned>(p.seqs_per_bias)] : p.beta_bias;
}
#endif
int efla_launch(const EflaParams& p, cudaStream_t stream);
extern int g_efla_chunked;
// Whole sequences from a zero state, any head_dim (efla_seq.cu).
bool efla_seq_applies(const EflaParams& p);
int efla_seq_launch(const EflaParams& p, cudaStream_t stream);
// Whole sequences of up to 128 tokens with half inputs and output, heads of 64 (efla_tc.cu).
bool efla_tc_applies(const EflaParams& p);
int efla_tc_launch(const EflaParams& p, bool early, int dev, int sms, cudaStream_t stream);

// Rank-r noise sums Z of a table of matrices in one launch (es_kernels.cu).
struct ZLowrankDesc {
    const int8_t* A;  // [pairs][rows][rank]
    long long A_ps;
    const int8_t* B;  // [pairs][rank][cols]
    long long B_ps;
    float* Z;         // [rows][cols]
    int rows, cols;
    int tile0;        // first 32 x 64 tile of this matrix in an unsharded launch over the table
};
inline int z_lowrank_tiles(int rows, int cols) { return ((rows + 31) / 32) * ((cols + 63) / 64); }
struct ZDenseDesc {
    uint64_t salt;
    const int8_t* noise;  // the step's noise [pair][n] in memory, for the table form
    long long zoff;
    int n;
    int rows;  // of a matrix: sharded by rows when they divide; 0 for a vector: sharded when it is long enough
};
__host__ __device__ inline void z_dense_range(const ZDenseDesc& d, int shard, int nshards, int& i0, int& cnt) {
    const bool split = nshards > 1 && (d.rows > 0 ? d.rows >= nshards && d.rows % nshards == 0 : d.n >= 4096 && d.n % nshards == 0);
    cnt = split ? d.n / nshards : d.n;
    i0 = split ? shard * cnt : 0;
}
// Tensors whose Z is formed from noise tables in the same launch (all have `noise` set, for all pairs).
struct ZTables {
    const ZDenseDesc* descs = nullptr;  // device
    int ndesc = 0;
    int blocks = 0;  // set by the launcher
    float* z_all = nullptr;
};
int z_lowrank_launch(const float* pair_weights, const ZLowrankDesc* d_descs, const ZLowrankDesc* h_descs, int ndesc, int pairs, int rank,
                     float cscale, int shard, int nshards, ZTables tables, const ZDenseDesc* h_tables, cudaStream_t stream);

// Apply phase of the ES update over a table of tensors (es_kernels.cu). The table does not change during a model's life: Z is given by
// an offset into the launch's Z buffer.
struct UpdApplyDesc {
    int8_t* w;       // ternary weights (nullptr for an fp32 vector)
    float* target;   // fp32 shadow of a matrix, or the vector itself
    float* ema;      // the tensor's RMS-EMA slot
    uint8_t* codes;  // NVFP4 copy of the weights (nullptr: none), row `row0` of its operand onwards
    uint8_t* sf;
    long long zoff;  // floats
    int n;
    int cols;        // of a matrix with an NVFP4 copy (a multiple of 16)
    int row0;        // first row inside the stacked operand
    int scaled;      // 1: the row scale of the stacked projection is folded into the scale bytes (second half of the quantiser table)
    int block0;      // first 256-element block of this tensor in the sum-of-squares launch
    int ublock0;     // first 1024-element block in the update launch
};
// tab: {1 / scale, scale byte} per block maximum, 128 entries unscaled and 128 with the row scale (update_quant_table).
// `up` (a power of two) is multiplied into the scale bytes only; whoever multiplies with the weights divides alpha by it.
void update_quant_table(float row_scale, float up, uint2 (&tab)[256]);
int update_apply_batched(const UpdApplyDesc* d_descs, int ndesc, int total_blocks, int total_ublocks, const float* z_all, const uint2* tab, float* partial,
                         float* inv_rms, int use_adaptive, float beta, float eps, float lr, float thresh, cudaStream_t stream);
// The NVFP4 copies alone, from the present weights.
int requantize_batched(const UpdApplyDesc* d_descs, int ndesc, int total_ublocks, const uint2* tab, cudaStream_t stream);

// Dense-noise Z of a table of tensors in one launch, from the hash.
int z_dense_table_launch(const float* pair_weights, const uint64_t* pair_seeds, const ZDenseDesc* d_descs, const ZDenseDesc* h_descs, int ndesc, int pairs,
                         int use_clt, int clt_k, int shard, int nshards, float* z_all, cudaStream_t stream);

// Fitness shaping of all pairs on the device, from the losses of their members (es_kernels.cu).
bool shape_fitness_applies(int pairs, int mode);
int shape_fitness_launch(const float* losses, int pairs, int mode, float clip, float* weights, cudaStream_t stream);

// Mean cross-entropy of every member (es_kernels.cu). partial: kCePartials floats per member (16 without counters). counters: one zeroed word per
// member, zero again afterwards; nullptr: the 16 group sums of every member only.
constexpr int kCePartials = 128;
int cross_entropy_launch(const float* logits, int ld, const float* bias, const int8_t* bias_noise, float sigma, const uint8_t* targets, int vocab, int members,
                         int rows_per_member, float* partial, unsigned* counters, float* loss_mean, cudaStream_t stream);

void count_launch();

}  // namespace bnf4
