// Block-scaled FP4 (NVFP4: e2m1 data, one ue4m3 scale per 16 K-elements) GEMM for sm_100a.
//
//   D[m,n] = alpha * sum_kb sfa[m,kb] * sfb[n,kb] * sum_{k in kb} a[m,k] * b[n,k]  (+ beta * C[m,n])
//            (+ s_member * sum_r t[m][g*rank+r] * A_pair[n][r])                      rank-r perturbation
//
// replaces the reference's CUTLASS Sm120 kernel behind gemm_ternary_f_nvfp4 /
// gemm_ternary_f_nvfp4_gelu_i8 (reference: src/cuda_kernels.cu:3145-3310, 4342-4607) and fuses the
// rank-r term of gemm_lora_f_kernel (reference: src/cuda_kernels.cu:1271-1305) into the tile epilogue.
//
// Structure of one CTA (128 x 128 output tiles, 576 threads):
//   warp 0      producer: TMA tiles of A and B (128 rows x 128 bytes = 256 K-elements, 128B swizzle) and
//               bulk copies of the matching scale-factor atoms into a ring of shared-memory stages
//   warp 1      owns TMEM; per stage copies the scale atoms to TMEM (tcgen05.cp 32x128b.warpx4) and issues
//               tcgen05.mma.kind::mxf4nvf4.block_scale (M128 x N128 x K64) accumulating fp32 in TMEM
//   warps 2..17 epilogue: tcgen05.ld the accumulator (four warps per TMEM lane quadrant, 32 columns each), apply
//               alpha/beta/rank-r/GELU, and store (TMA store through swizzled staging, or direct)
// The kernel is persistent (one CTA per SM, tiles assigned round-robin): the producer runs up to four k-blocks
// ahead (long K: CTA pairs on 256 x 256 tiles, see PAIR below), and two TMEM accumulators let the MMAs of tile i+1 overlap the epilogue of tile i. Every mbarrier wait is bounded: on expiry the kernel records an error
// word, leaves its role loop, frees TMEM and returns.

#include <cuda.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"

namespace bnf4 {

namespace {

constexpr int BM = 128;             // tile rows
constexpr int BN = 128;             // tile columns
constexpr int BK = 256;             // K elements per stage (128 bytes of packed e2m1 per row)
constexpr int UMMA_K = 64;          // K elements per tcgen05.mma
constexpr int kStages = 4;
constexpr int kStageABytes = BM * 128;
constexpr int kStageBBytes = BN * 128;
constexpr int kStageSfBytes = 4 * 512;  // four 128-row x 64-K atoms
constexpr int kEpiWarps = 16;
constexpr int kEpiBufBytes = 32 * 32 * 4;  // one 32 x 32 fp32 box
constexpr int kThreads = 64 + kEpiWarps * 32;
constexpr int kTmemCols = 512;      // two 128-column accumulators + kStages * 32 scale columns, rounded to a power of two
constexpr int kAccCol = 0;
constexpr int kSfCol = 256;

constexpr int kSmemA = 0;
constexpr int kSmemB = kSmemA + kStages * kStageABytes;
constexpr int kSmemSfa = kSmemB + kStages * kStageBBytes;
constexpr int kSmemSfb = kSmemSfa + kStages * kStageSfBytes;
constexpr int kSmemEpi = kSmemSfb + kStages * kStageSfBytes;
constexpr int kSmemLora = kSmemEpi + kEpiWarps * kEpiBufBytes;
constexpr int kSmemBar = kSmemLora + kEpiWarps * 4 * 32 * 4;  // per epilogue warp: [4][32] floats of the pair's A factor
constexpr int kSmemTotal = kSmemBar + 128;
constexpr int kSmemAlloc = kSmemTotal + 1024;  // slack for manual 1024-byte alignment

// CTA-pair instances (PAIR): two CTAs of a cluster share one 256 x 256 tile. Per stage a CTA holds its 128 rows of A, its half of
// the 256 B rows, the scale atoms of its A rows and those of all 256 B rows.
constexpr int kPairStageBBytes = 2 * 64 * 128;
constexpr int kPairStageSfbBytes = 2 * kStageSfBytes;
constexpr int kPairSmemSfa = kSmemB + kStages * kPairStageBBytes;
constexpr int kPairSmemSfb = kPairSmemSfa + kStages * kStageSfBytes;
constexpr int kPairSmemEpi = kPairSmemSfb + kStages * kPairStageSfbBytes;
constexpr int kPairSmemLora = kPairSmemEpi + kEpiWarps * kEpiBufBytes;
constexpr int kPairSmemBar = kPairSmemLora + kEpiWarps * 4 * 32 * 4;
constexpr int kPairSmemAlloc = kPairSmemBar + 128 + 1024;
constexpr int kPairAcc = 3;                 // accumulator blocks of 128 columns: even tiles fill the first two, odd ones the last two
constexpr int kPairSfCol = kPairAcc * 128;  // two scale slots of 16 (A) + 32 (B) columns behind them
static_assert(kPairSmemAlloc <= 232448 && kSmemAlloc <= 232448, "shared memory of one SM");

}  // namespace
int g_gemm_allow_tma_store = 1;  // host toggle: 0 forces the direct-store epilogue
namespace {

// Instruction descriptor of kind::mxf4nvf4 (block-scaled): a/b format e2m1 (=1) at bits 7 and 10,
// K-major A and B, N>>3 at bit 17, ue4m3 scales (bit 23 = 0), M>>4 at bit 24, scale ids 0, dense K = 64.
constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>(BM >> 4) << 24);

constexpr uint32_t kIdescPairM = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(2 * BM >> 4) << 24);                 // M 256 ...
constexpr uint32_t kIdescPair256 = kIdescPairM | (256u >> 3 << 17), kIdescPair128 = kIdescPairM | (128u >> 3 << 17);  // ... x N 256 / N 128

// Scale atoms as rows of 512 bytes (the pair instances fetch them with tiled copies, which can signal the leading CTA's barrier).
struct PairMaps {
    CUtensorMap sfa, sfb;
};
struct B2Map {
    CUtensorMap b2;  // the second B operand (GemmParams::b2)
};
struct NoMaps {};
template <bool PAIR, bool B2>
using ExtraMaps = std::conditional_t<PAIR, PairMaps, std::conditional_t<B2, B2Map, NoMaps>>;

struct KernelArgs {
    GemmParams p;
    int use_tma_store;
    int k_atoms;  // scale atoms along K
    uint32_t group_magic;  // ceil(2^32 / group_cols) (0 when group_cols == 0)
    uint32_t rpm_magic;    // floor(2^32 / rows_per_member), at most 2^32 - 1
    const uint8_t* lut;  // table of the block quantiser (EPI_GELU_FP4)
    int total_tiles;
    int ks_wrap;  // K blocks after which A starts again and B2 follows B (0: no second operand)
    int n_tiles;  // tiles along N (of 256 columns in the pair instances); blockIdx.x = m_tile * n_tiles + n_tile (N fastest: CTAs that share A rows run together)
    // A CTA's (or pair's) first tile and the way to its next one without a division: four of them stood between the predecessor's end and the first load (800
    // cycles; a GEMM of one tile behind another 4.7 -> 4.3 us).
    uint32_t tile_magic;  // ceil(2^32 / n_tiles): exact quotients for the few hundred CTAs (0: one tile along N)
    int step_n, step_m;   // CTAs (pairs) of the grid % and / n_tiles
};

// Persistent kernel: one CTA per SM walks the tile list (tile = m_tile * n_tiles + n_tile, N fastest so that
// CTAs working at the same time share rows of A through L2). Three roles run concurrently on different tiles:
// the producer prefetches operands up to kStages k-blocks ahead, the MMA warp fills one of two TMEM
// accumulators while the sixteen epilogue warps drain the other one.
// RK: the form of the rank term. 0 = none; 1 = the batched driver's common case (rank 1, no C operand, every 128-row tile inside one member), which
// carries none of the general paths; 3 and 5 = rank 2 and 4 whose pairs start at multiples of 32 rows, so that a warp's rows share a pair; 2 and 4 =
// every other one of rank 1 and 2, 3 and 4, with zeros for a factor that is not there. The number of products is thereby known to the compiler: one
// instance tested the rank inside the loop over the columns (and spilled: 88 and 114 bytes with FP4 output, 4 to 28 with the others). Figures, one such instance -> these, us: 88800 x 320 x 320 rank 2 residual 44 -> 32,
// 88800 x 961 x 320 rank 2 halves 69 -> 52, 88800 x 960 x 320 GELU to FP4 rank 2 141 -> 106, rank 3 with members of 1100 rows 152 -> 132, 65536 x 512 x 2048 rank 2
// residual 65 -> 46, 16384 x 512 x 512 rank 3 fp32 11.9 -> 10.8. Without forms 3 and 5 those of rank 2 and 4 lose 2 to 12 % (33.5, 54, 119). 16384 x 4096 x 4096 rank 3 fp32
// stands at 132 to 150 with either (one build's runs differ by 5 % there; an instance of three products gave nothing), the other epilogues gain: 150 -> 144, 125 -> 121, 154 -> 146. (262144 x 1024 x 512 with GELU to FP4 and no rank term: 303 us as a case of a general instance, 256 us.)
// B2: the instance with a second B operand (no rank term); the others carry no tests for one (a rank-2 term with GELU to FP4 446 -> 412 us).
// PAIR: the instance for operands with many K blocks. On the in-order pipe a scale copy costs about 44 cycles and an M 128 x N 128 MMA
// 64 (measured, one CTA): 8 copies and 4 MMAs per 256-element K block of a 128 x 128 tile take 560 cycles before any operand
// traffic, 860 with it. A CTA pair (cta_group::2) on a 256 x 256 tile needs 12 copies and 4 MMAs of N 256 for four times the work; the
// long MMAs hide most of the copies: 718 cycles (968 with twice as many N 128 MMAs), and each CTA loads 38 instead of 68 KB.
// There each K step's copies stand directly in front of its MMA: behind the MMA of the step before they run under it, while twelve in a row in front of four
// MMAs do not (262144 x 1024 x 4096, rank 1, residual epilogue 540 -> 494 us; 16384 x 4096 x 4096, rank 4, 164.7 -> 157.5). A single CTA's N 128 MMAs are
// too short for that: eight copies in a row overlap one another better (262144 x 1537 x 512 205 us, 213 with the copies in between; 48 small GEMMs of a token step 239.5, 242).
// Accumulators: even tiles use the 128-column blocks 0 and 1, odd tiles 1 and 2, and the epilogue drains block 1 first, so that the
// next tile starts as soon as the shared block has been read. The epilogue code sees a sequence of 128 x 128 sub-tiles.
template <int EPI, int RK, bool PAIR, bool B2>
__global__ void __launch_bounds__(kThreads, 1) gemm_nvfp4_kernel(const __grid_constant__ CUtensorMap map_a,
                                                                 const __grid_constant__ CUtensorMap map_b,
                                                                 const __grid_constant__ CUtensorMap map_d,
                                                                 const __grid_constant__ ExtraMaps<PAIR, B2> maps_sf,
                                                                 const KernelArgs args) {
    constexpr int kAcc = PAIR ? kPairAcc : 2;  // TMEM accumulators
    constexpr int oSmemEpi = PAIR ? kPairSmemEpi : kSmemEpi, oSmemLora = PAIR ? kPairSmemLora : kSmemLora, oSmemBar = PAIR ? kPairSmemBar : kSmemBar;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

    const GemmParams& p = args.p;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int num_ks = ((p.k + BK - 1) / BK) << (B2 ? 1 : 0);  // K blocks of a tile (both B operands)
    const int total_tiles = args.total_tiles;

    const uint32_t bar_full = smem_base + oSmemBar;               // kStages x 8 bytes (PAIR: the leading CTA's count for both)
    const uint32_t bar_empty = bar_full + 8 * kStages;            // kStages x 8 bytes
    const uint32_t bar_acc_full = bar_empty + 8 * kStages;        // kAcc x 8 bytes
    const uint32_t bar_acc_empty = bar_acc_full + 8 * kAcc;       // kAcc x 8 bytes (PAIR: likewise)
    const uint32_t tmem_slot = bar_acc_empty + 8 * kAcc;          // 4 bytes
    volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + oSmemBar + 16 * kStages + 16 * kAcc);
    uint32_t rank = 0;  // of this CTA in its pair
    if constexpr (PAIR) rank = cluster_rank();
    // the tiles this CTA (or pair) walks: unit, unit + units, ..
    const unsigned unit = PAIR ? blockIdx.x >> 1 : blockIdx.x, units = PAIR ? gridDim.x >> 1 : gridDim.x;
    const int first_m = static_cast<int>(args.tile_magic == 0 ? unit : __umulhi(unit, args.tile_magic)), first_n = static_cast<int>(unit) - first_m * args.n_tiles;

    if (threadIdx.x == 64) {  // the tensor maps come from the parameter area: fetch them before the predecessor has finished
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
        if (args.use_tma_store) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_d)) : "memory");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (int b = 0; b < kAcc; ++b) {
            mbar_init(bar_acc_full + 8 * b, 1);
            mbar_init(bar_acc_empty + 8 * b, PAIR ? 2 * kEpiWarps : kEpiWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (PAIR) {
            tmem_alloc_pair(tmem_slot, kTmemCols);
            tmem_relinquish_pair();
        } else {
            tmem_alloc(tmem_slot, kTmemCols);
            tmem_relinquish();
        }
    }
    tc_fence_before();
    if constexpr (PAIR) cluster_sync();  // the peer's barriers exist before anything signals them
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_gen;
    pdl_wait();  // the set-up above overlaps the predecessor's tail; everything below reads what it wrote

    if (PAIR && warp == 0) {
        // ------------------------------ producer of one half of a pair ------------------------------
        if constexpr (PAIR) {
            int kc = 0, s = 0;
            uint32_t empty_parity = 1;
            bool ok = true;
            int mt = first_m, nt = first_n;
            for (unsigned tile = unit; tile < static_cast<unsigned>(total_tiles) && ok; tile += units) {
                const bool two = nt * 256 + 128 < p.n;  // the second half has columns
                // each CTA holds half of the B rows of the pair's MMA: 128 of 256, or 64 of 128
                const int my = mt * 256 + static_cast<int>(rank) * BM, ny = nt * 256 + static_cast<int>(rank) * (two ? 128 : 64);
                const int sfa_row = (my >> 7) * args.k_atoms, sfb_row = nt * 2 * args.k_atoms;
                const uint32_t bytes = 2u * (kStageABytes + kStageSfBytes + (two ? 2u : 1u) * (64 * 128 + kStageSfBytes));
                for (int ks = 0; ks < num_ks; ++ks, ++kc) {
                    if (kc >= kStages) {
                        ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, empty_parity, 1));
                        if (!ok) break;
                    }
                    if (elect_one()) {
                        const uint32_t bar = map_to_leader(bar_full + 8 * s);
                        if (rank == 0) mbar_expect_tx(bar_full + 8 * s, bytes);
                        tma_load_2d_pair(smem_base + kSmemA + s * kStageABytes, &map_a, ks * 128, my, bar);
                        tma_load_2d_pair(smem_base + kSmemB + s * kPairStageBBytes, &map_b, ks * 128, ny, bar);
                        tma_load_2d_pair(smem_base + kPairSmemSfa + s * kStageSfBytes, &maps_sf.sfa, 0, sfa_row + 4 * ks, bar);
                        tma_load_2d_pair(smem_base + kPairSmemSfb + s * kPairStageSfbBytes, &maps_sf.sfb, 0, sfb_row + 4 * ks, bar);
                        if (two) {
                            tma_load_2d_pair(smem_base + kSmemB + s * kPairStageBBytes + 64 * 128, &map_b, ks * 128, ny + 64, bar);
                            tma_load_2d_pair(smem_base + kPairSmemSfb + s * kPairStageSfbBytes + kStageSfBytes, &maps_sf.sfb, 0, sfb_row + args.k_atoms + 4 * ks, bar);
                        }
                    }
                    __syncwarp();
                    if (++s == kStages) { s = 0; empty_parity ^= 1u; }
                }
                nt += args.step_n;
                mt += args.step_m;
                if (nt >= args.n_tiles) { nt -= args.n_tiles; ++mt; }
            }
            // the last stages' releases arrive from the leading CTA: wait for them, so that none is in flight towards a CTA that has left
            for (int i = 0; i < min(kc, kStages) && ok; ++i) {
                if (kc < kStages) ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * i, 0, 1));
                else {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, empty_parity, 1));
                    if (++s == kStages) { s = 0; empty_parity ^= 1u; }
                }
            }
        }
    } else if (PAIR && warp == 1) {
        // ------------------------------ MMA issuer: the leading CTA's warp works for both ------------------------------
        if constexpr (PAIR) {
            const uint64_t adesc0 = smem_desc(smem_base + kSmemA, 16, 1024, kLayoutSw128);
            const uint64_t bdesc0 = smem_desc(smem_base + kSmemB, 16, 1024, kLayoutSw128);
            const uint64_t sfadesc0 = smem_desc(smem_base + kPairSmemSfa, 0, 128, kLayoutNone);
            const uint64_t sfbdesc0 = smem_desc(smem_base + kPairSmemSfb, 0, 128, kLayoutNone);
            int s = 0;
            uint32_t full_parity = 0, kc = 0, odd = 0;
            uint32_t empty_par = 0, used = 0;  // per accumulator block (bit): parity of the drain to wait for next; whether it was used before
            bool ok = rank == 0;
            int nt = first_n;
            for (unsigned tile = unit; tile < static_cast<unsigned>(total_tiles) && ok; tile += units, odd ^= 1u) {
                const bool two = nt * 256 + 128 < p.n;
                // both CTAs' epilogues must have drained the blocks
                for (uint32_t b = odd; b <= odd + (two ? 1u : 0u) && ok; ++b) {
                    if ((used >> b) & 1u) {
                        ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_empty + 8 * b, (empty_par >> b) & 1u, 4));
                        empty_par ^= 1u << b;
                    }
                    used |= 1u << b;
                }
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc = tmem_base + odd * 128, idesc = two ? kIdescPair256 : kIdescPair128;
                for (int ks = 0; ks < num_ks; ++ks, ++kc) {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * s, full_parity, 2));
                    if (!ok) break;
                    tc_fence_after();
                    const int nk = min(4, (p.k - ks * BK) / UMMA_K);
                    const uint32_t t_sfa = tmem_base + kPairSfCol + (kc & 1u) * 48, t_sfb = t_sfa + 16;  // the pipe is in order: two slots suffice
                    const uint64_t sfa_d = sfadesc0 + static_cast<uint64_t>(s * (kStageSfBytes >> 4)), sfb_d = sfbdesc0 + static_cast<uint64_t>(s * (kPairStageSfbBytes >> 4));
                    const uint64_t a_d = adesc0 + static_cast<uint64_t>(s * (kStageABytes >> 4)), b_d = bdesc0 + static_cast<uint64_t>(s * (kPairStageBBytes >> 4));
                    if (elect_one()) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (j < nk) {
                                tc_cp_sf_pair(t_sfa + 4 * j, sfa_d + static_cast<uint64_t>(j * (512 >> 4)));
                                tc_cp_sf_pair(t_sfb + 8 * j, sfb_d + static_cast<uint64_t>(j * (512 >> 4)));
                                if (two) tc_cp_sf_pair(t_sfb + 8 * j + 4, sfb_d + static_cast<uint64_t>((kStageSfBytes + j * 512) >> 4));
                                const uint64_t kj = static_cast<uint64_t>(j * (32 >> 4));
                                tc_mma_nvf4_pair(acc, a_d + kj, b_d + kj, idesc, t_sfa + 4 * j, t_sfb + 8 * j, ks > 0 || j > 0 ? 1u : 0u);
                            }
                        }
                        tc_commit_pair(bar_empty + 8 * s);
                        if (ks == num_ks - 1) {
                            tc_commit_pair(bar_acc_full + 8 * odd);
                            if (two) tc_commit_pair(bar_acc_full + 8 * odd + 8);
                        }
                    }
                    __syncwarp();
                    if (++s == kStages) { s = 0; full_parity ^= 1u; }
                }
                nt += args.step_n;
                if (nt >= args.n_tiles) nt -= args.n_tiles;
            }
        }
    } else if (warp == 0) {
        // ------------------------------ producer ------------------------------
        {
            // running indices instead of divisions, addresses advanced by constants
            int kc = 0;  // k-block counter across tiles
            int s = 0;
            uint32_t empty_parity = 1;  // parity of the phase that precedes the first completion: the first pass does not wait
            bool ok = true;
            const int step_n = args.step_n, step_m = args.step_m;
            int m_tile = first_m - step_m;
            int n_tile = first_n - step_n;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                n_tile += step_n;
                m_tile += step_m;
                if (n_tile >= args.n_tiles) { n_tile -= args.n_tiles; ++m_tile; }
                const uint8_t* sfa_src = static_cast<const uint8_t*>(p.sfa) + static_cast<size_t>(m_tile) * args.k_atoms * 512;
                const uint8_t* sfb_src = static_cast<const uint8_t*>(p.sfb) + static_cast<size_t>(n_tile) * args.k_atoms * 512;
                const int my = m_tile * BM, ny = n_tile * BN;
                int atoms_left = args.k_atoms, x = 0, by = ny;
                const CUtensorMap* bmap = &map_b;
                for (int ks = 0; ks < num_ks; ++ks, ++kc, x += 128) {
                    if constexpr (B2) {
                        if (ks == args.ks_wrap) {
                            const int member = my / p.rows_per_member;
                            x = 0;
                            by = member * p.b2_rows + ny;
                            bmap = &maps_sf.b2;
                            atoms_left = args.k_atoms;
                            sfa_src = static_cast<const uint8_t*>(p.sfa) + static_cast<size_t>(m_tile) * args.k_atoms * 512;
                            sfb_src = static_cast<const uint8_t*>(p.sfb2) + static_cast<size_t>(by >> 7) * args.k_atoms * 512;
                        }
                    }
                    if (kc >= kStages) {
                        ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, empty_parity, 1));
                        if (!ok) break;
                    }
                    const uint32_t sf_bytes_stage = static_cast<uint32_t>(min(4, atoms_left)) * 512u;
                    atoms_left -= 4;
                    const uint32_t bar = bar_full + 8 * s;
                    if (elect_one()) {
                        mbar_expect_tx(bar, kStageABytes + kStageBBytes + 2 * sf_bytes_stage);
                        tma_load_2d(smem_base + kSmemA + s * kStageABytes, &map_a, x, my, bar);
                        tma_load_2d(smem_base + kSmemB + s * kStageBBytes, bmap, x, by, bar);
                        bulk_load_1d(smem_base + kSmemSfa + s * kStageSfBytes, sfa_src, sf_bytes_stage, bar);
                        bulk_load_1d(smem_base + kSmemSfb + s * kStageSfBytes, sfb_src, sf_bytes_stage, bar);
                    }
                    __syncwarp();
                    sfa_src += 2048;
                    sfb_src += 2048;
                    if (++s == kStages) { s = 0; empty_parity ^= 1u; }
                }
            }
            pdl_trigger();  // every operand is on its way: what is left of this CTA is its last tile
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        {
            // The issue rate of this role bounds the mainloop (it shares an issue port with four busy epilogue warps), so the loop
            // is kept lean: descriptors are a stage-0 constant plus a stage / K-step increment of the 14-bit start-address field
            // (bytes >> 4), and the four K-steps of a full stage are unrolled.
            const uint64_t adesc0 = smem_desc(smem_base + kSmemA, 16, 1024, kLayoutSw128);
            const uint64_t bdesc0 = smem_desc(smem_base + kSmemB, 16, 1024, kLayoutSw128);
            const uint64_t sfadesc0 = smem_desc(smem_base + kSmemSfa, 0, 128, kLayoutNone);
            const uint64_t sfbdesc0 = smem_desc(smem_base + kSmemSfb, 0, 128, kLayoutNone);
            int kc = 0, it = 0;
            int s = 0;
            uint32_t full_parity = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++it) {
                const int buf = it & 1;
                if (it >= 2) {  // the epilogue must have drained this accumulator (tile it-2)
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_empty + 8 * buf, ((it >> 1) - 1) & 1, 4));
                    if (!ok) break;
                    tc_fence_after();
                }
                const uint32_t acc_col = tmem_base + kAccCol + buf * BN;
                for (int ks = 0; ks < num_ks; ++ks, ++kc) {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * s, full_parity, 2));
                    if (!ok) break;
                    tc_fence_after();
                    const int nk = min(4, (p.k - (B2 && ks >= args.ks_wrap ? ks - args.ks_wrap : ks) * BK) / UMMA_K);
                    const uint32_t t_sfa = tmem_base + kSfCol + s * 32;
                    const uint32_t t_sfb = t_sfa + 16;
                    const uint64_t sfa_d = sfadesc0 + static_cast<uint64_t>(s * (kStageSfBytes >> 4));
                    const uint64_t sfb_d = sfbdesc0 + static_cast<uint64_t>(s * (kStageSfBytes >> 4));
                    const uint64_t a_d = adesc0 + static_cast<uint64_t>(s * (kStageABytes >> 4));
                    const uint64_t b_d = bdesc0 + static_cast<uint64_t>(s * (kStageBBytes >> 4));
                    if (elect_one()) {
                        if (nk == 4) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                tc_cp_sf(t_sfa + 4 * j, sfa_d + static_cast<uint64_t>(j * (512 >> 4)));
                                tc_cp_sf(t_sfb + 4 * j, sfb_d + static_cast<uint64_t>(j * (512 >> 4)));
                            }
                            tc_mma_nvf4(acc_col, a_d, b_d, kIdesc, t_sfa, t_sfb, ks > 0 ? 1u : 0u);
#pragma unroll
                            for (int j = 1; j < 4; ++j)
                                tc_mma_nvf4(acc_col, a_d + static_cast<uint64_t>(j * (32 >> 4)), b_d + static_cast<uint64_t>(j * (32 >> 4)), kIdesc,
                                            t_sfa + 4 * j, t_sfb + 4 * j, 1u);
                        } else {
                            for (int j = 0; j < nk; ++j) {
                                tc_cp_sf(t_sfa + 4 * j, sfa_d + static_cast<uint64_t>(j * (512 >> 4)));
                                tc_cp_sf(t_sfb + 4 * j, sfb_d + static_cast<uint64_t>(j * (512 >> 4)));
                            }
                            for (int j = 0; j < nk; ++j)
                                tc_mma_nvf4(acc_col, a_d + static_cast<uint64_t>(j * (32 >> 4)), b_d + static_cast<uint64_t>(j * (32 >> 4)), kIdesc,
                                            t_sfa + 4 * j, t_sfb + 4 * j, (ks > 0 || j > 0) ? 1u : 0u);
                        }
                        tc_commit(bar_empty + 8 * s);  // frees this smem stage once the MMAs above have read it
                        if (ks == num_ks - 1) tc_commit(bar_acc_full + 8 * buf);  // accumulator of this tile complete
                    }
                    __syncwarp();
                    if (++s == kStages) { s = 0; full_parity ^= 1u; }
                }
            }
        }
    } else {
        // ------------------------------ epilogue: 16 warps, four per TMEM lane quadrant, 32 columns each ------------------------------
        const int ew = warp - 2;   // 0..15
        const int q = warp & 3;    // TMEM lane quadrant this warp may access
        const int c = ew >> 2;     // 32-column chunk of the tile handled by this warp
        const uint32_t epi_buf = smem_base + oSmemEpi + ew * kEpiBufBytes;
        uint8_t* epi_gen = smem_gen + oSmemEpi + ew * kEpiBufBytes;
        bool ok = true;
        int it = 0;
        int stage_half = 0;  // EPI_F16: which half of the staging buffer the next store uses
        if constexpr (EPI == EPI_GELU_FP4) {
            // The block quantiser's table ({1 / scale, scale byte} per amax, 1 KB) lives in the staging area the fp32 epilogue would use.
            if (ew * 32 + lane < 128)
                reinterpret_cast<uint2*>(smem_gen + oSmemEpi)[ew * 32 + lane] =
                    __ldg(reinterpret_cast<const uint2*>(args.lut + kQuantBlockTabOffset) + ew * 32 + lane);
            asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        }
        // RK 2 and up with FP4 output: the vectors of the next projection, fetched a tile ahead like the factors (loads where they are used left the warps waiting: 65536 x 8192
        // x 2048 with four of them 883 -> 878 us), and a place where the rows' sums are turned round (128-byte atomics instead of sixteen sectors each: 787 us).
        constexpr bool kInside = RK == 3 || RK == 5, kStageNext = RK >= 2 && EPI == EPI_GELU_FP4;
        constexpr int kTerms = RK >= 4 ? 4 : 2;  // products of the rank term (factors that are not there are zeros)
        int4* next_sh = reinterpret_cast<int4*>(smem_gen + oSmemEpi + kQuantBlockTabBytes + ew * 640);  // [4][32] bytes, then [32][4] sums
        // Perturbation context of one tile: this thread's row (projections t, sign, pair) and this thread's element of the A factor
        // of the warp's first pair for the tile's columns. It is fetched one tile ahead so that the global-load latency hides
        // behind the previous tile's epilogue. A warp whose 32 rows reach into the next pair (members that are no multiple of the tile
        // height) applies the pairs one after the other, each to its own rows.
        struct LoraCtx {
            int member;
            int tr[4];    // raw integers: converted to float only when the tile is processed, so that nothing waits
            int aval[4];  // on these loads earlier;  aval[r] = A[pair of the warp's first row][col0 + lane][r]
            int next_b;   // RK 2 and up: this thread's word of the pair's vectors of the next projection: vector lane / 8, columns col0 + 4 (lane % 8) ..
        };
        const int row_in_tile = q * 32 + lane;
        // Tile coordinates advance by additions (tiles are walked in steps of gridDim.x): no division per tile.
        const int step_n = args.step_n, step_m = args.step_m;
        // m_tile counts 128-row tiles (of a pair's tile: this CTA's), n_tile 128-column tiles; the halves of a pair's tile follow each other.
        // PAIR: `odd` = parity of the tile, `last` = no further half follows in this tile.
        struct TileIdx { int m_tile, n_tile, odd; bool last; };
        auto first_half = [&](TileIdx& t, int nt) {  // of tile column nt: the half in the shared accumulator block
            const bool two = nt * 256 + 128 < p.n;
            t.n_tile = 2 * nt + (two && t.odd == 0 ? 1 : 0);
            t.last = !two;
        };
        auto advance = [&](TileIdx& t) {
            if constexpr (PAIR) {
                if (!t.last) { t.n_tile ^= 1; t.last = true; return; }
                int nt = (t.n_tile >> 1) + step_n;
                t.m_tile += 2 * step_m;
                if (nt >= args.n_tiles) { nt -= args.n_tiles; t.m_tile += 2; }
                t.odd ^= 1;
                first_half(t, nt);
            } else {
                t.n_tile += step_n;
                t.m_tile += step_m;
                if (t.n_tile >= args.n_tiles) { t.n_tile -= args.n_tiles; ++t.m_tile; }
            }
        };
        const int m_end = PAIR ? 2 * (total_tiles / args.n_tiles) : 0;  // first 128-row tile behind the matrix, pairs rounded up
        auto in_range = [&](const TileIdx& t) { return t.m_tile < m_end; };
        // a pair's second CTA may have no rows left in the last tile: it has nothing to fetch then
        auto has_rows = [&](const TileIdx& t) { return t.m_tile < m_end && t.m_tile * BM < p.m; };
        // Members are visited in ascending order, so when tiles never straddle members (rows_per_member a multiple of the
        // tile height) the member of the next tile is tracked with comparisons instead of a division per row.
        int trk_member = static_cast<int>(opaque_zero());  // (the pair's vectors are loaded read-only: their addresses depend on this)
        long long trk_end = p.rows_per_member;  // first row of member trk_member + 1
        const uint32_t group_magic = args.group_magic;  // ceil(2^32 / group_cols): exact quotients for columns below 65536
        auto member_of = [&](unsigned row) {  // row / rows_per_member: the multiply-high is exact or one too small
            if (p.rows_per_member <= 0) return 0;
            const unsigned e = __umulhi(row, args.rpm_magic);
            return static_cast<int>(row - e * static_cast<unsigned>(p.rows_per_member) >= static_cast<unsigned>(p.rows_per_member) ? e + 1 : e);
        };
        const int terms = kInside ? kTerms : p.rank;
        auto load_a = [&](int pr, int n, int (&aval)[4]) {
            const int8_t* Ag = p.lora_A + static_cast<size_t>(pr) * p.lora_A_pair_stride + static_cast<size_t>(n) * terms;
#pragma unroll
            for (int r = 0; r < kTerms; ++r) aval[r] = r < terms ? Ag[r] : 0;
        };
        auto fetch_ctx = [&](const TileIdx& t, bool valid, LoraCtx& cx) {
            cx.member = 0;
            cx.tr[0] = cx.tr[1] = cx.tr[2] = cx.tr[3] = 0;
            cx.aval[0] = cx.aval[1] = cx.aval[2] = cx.aval[3] = 0;
            if (!valid) return;
            const int m0_ = t.m_tile * BM, col0_ = t.n_tile * BN + c * 32;
            const int row_ = m0_ + row_in_tile;  // (rows fit 31 bits: p.m is an int)
            cx.member = member_of(static_cast<unsigned>(min(row_, p.m - 1)));  // (rows past m are never stored)
            if (row_ < p.m && col0_ < p.n) {
                const int g = p.group_cols > 0 ? static_cast<int>(__umulhi(static_cast<uint32_t>(col0_), group_magic)) : 0;
                const int* tp = p.lora_t + static_cast<size_t>(row_) * p.t_stride + g * terms;
#pragma unroll
                for (int r = 0; r < kTerms; ++r)
                    if (r < terms) cx.tr[r] = tp[r];
            }
            const int first = __shfl_sync(0xffffffffu, cx.member, 0) >> 1;
            if (col0_ + lane < p.n) load_a(first, col0_ + lane, cx.aval);
            if constexpr (kStageNext) {  // (n is a multiple of 32)
                if (col0_ < p.n && (lane >> 3) < p.next_nvec)
                    cx.next_b = *reinterpret_cast<const int*>(p.next_tvec + static_cast<size_t>(first) * p.next_tvec_pair_stride + static_cast<size_t>(lane >> 3) * p.n + col0_ + 4 * (lane & 7));
            }
        };
        // The common case (rank 1, tiles inside one member) with as few instructions as possible: this phase sits on the serial
        // path of every tile.
        constexpr bool R1 = RK == 1, R0 = RK == 0;
        const int* t_row = !R0 && p.rank > 0 ? p.lora_t + static_cast<size_t>(row_in_tile) * p.t_stride : nullptr;
        auto fetch_fast = [&](const TileIdx& t, bool valid, LoraCtx& cx) {
            cx.member = 0;
            cx.tr[0] = 0;
            cx.aval[0] = 0;
            if (!valid) return;
            const int m0_ = t.m_tile * BM, col0_ = t.n_tile * BN + c * 32;
            while (m0_ >= trk_end) { ++trk_member; trk_end += p.rows_per_member; }
            cx.member = trk_member;
            if ((R1 || m0_ + row_in_tile < p.m) && col0_ < p.n) {
                const int g = p.group_cols > 0 ? static_cast<int>(__umulhi(static_cast<uint32_t>(col0_), group_magic)) : 0;
                cx.tr[0] = t_row[static_cast<size_t>(m0_) * p.t_stride + g];
            }
            if (col0_ + lane < p.n) cx.aval[0] = __ldg(p.lora_A + static_cast<size_t>(trk_member >> 1) * p.lora_A_pair_stride + col0_ + lane);
        };
        TileIdx cur_t{first_m, first_n, 0, true};
        if constexpr (PAIR) {
            cur_t.m_tile = 2 * cur_t.m_tile + static_cast<int>(rank);
            first_half(cur_t, cur_t.n_tile);
        }
        TileIdx nxt_t = cur_t;
        // EPI_ADD_I8 through TMA: this warp's 32 x 32-byte box of the residual stream is loaded one tile ahead into one of
        // three 1 KB buffers (each with its own mbarrier), updated in place and stored from there. A lane-per-row access to
        // global memory touches 32 lines per instruction and kept the load/store unit busy for a third of the tile period.
        const bool res_tma = EPI == EPI_ADD_I8 && args.use_tma_store != 0;
        const uint32_t rbar = epi_buf + 3072;
        int rb_cur = 0, rb_last = 2;
        uint32_t r_par = 0;  // bit b: parity of the phase to wait for on buffer b
        bool have_cur = false, have_nxt = false;
        auto issue_res_load = [&](const TileIdx& t, bool valid) {
            const int col0_ = t.n_tile * BN + c * 32;
            have_nxt = valid && col0_ < p.n && (!R0 || t.m_tile * BM + q * 32 < p.m);
            if (!have_nxt) return;
            rb_last = rb_last == 2 ? 0 : rb_last + 1;
            if (lane == 0) {
                bulk_wait_read<1>();  // the store that last read this buffer (three tiles back) has left shared memory
                mbar_expect_tx(rbar + 8 * rb_last, 1024);
                tma_load_2d(epi_buf + rb_last * 1024, &map_d, col0_, t.m_tile * BM + q * 32, rbar + 8 * rb_last);
            }
        };
        if constexpr (EPI == EPI_ADD_I8) {
            if (res_tma) {
                if (lane == 0) {
                    mbar_init(rbar, 1);
                    mbar_init(rbar + 8, 1);
                    mbar_init(rbar + 16, 1);
                    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
                    fence_async_smem();
                }
                __syncwarp();
                issue_res_load(cur_t, PAIR ? has_rows(cur_t) : static_cast<int>(blockIdx.x) < total_tiles);
            }
        }
        LoraCtx nxt;
        nxt.tr[1] = nxt.tr[2] = nxt.tr[3] = 0;
        nxt.aval[1] = nxt.aval[2] = nxt.aval[3] = 0;
        nxt.next_b = 0;
        if constexpr (R0) nxt.member = 0;
        else if (R1) fetch_fast(cur_t, PAIR ? has_rows(cur_t) : static_cast<int>(blockIdx.x) < total_tiles, nxt);
        else fetch_ctx(cur_t, PAIR ? has_rows(cur_t) : static_cast<int>(blockIdx.x) < total_tiles, nxt);
        uint32_t pfull = 0;  // PAIR: parities of the completions to wait for (bit per accumulator block)
        uint32_t acc_empty_bar = bar_acc_empty;
        if constexpr (PAIR) acc_empty_bar = map_to_leader(bar_acc_empty);
        for (int tile = blockIdx.x; (PAIR ? in_range(nxt_t) : tile < total_tiles) && ok; tile += gridDim.x, ++it) {
            cur_t = nxt_t;
            const int buf = PAIR ? (cur_t.n_tile & 1) + cur_t.odd : it & 1;
            advance(nxt_t);
            const bool more = PAIR ? has_rows(nxt_t) : tile + static_cast<int>(gridDim.x) < total_tiles;
            const int m0 = cur_t.m_tile * BM, n0 = cur_t.n_tile * BN;
            const long long row = static_cast<long long>(m0) + row_in_tile;
            const bool row_ok = R1 || row < p.m;  // (the rank-1 instance runs with m a multiple of the tile height)
            const int col0 = n0 + c * 32;
            // warp-uniform: the warp's part of the tile lies in the matrix (rows: the few of a token step; with a rank term the test cost ragged members 2 %)
            const bool chunk_ok = col0 < p.n && (!R0 || m0 + q * 32 < p.m);

            const int member = nxt.member, pair = member >> 1;
            float tr[4] = {R0 ? 0.0f : static_cast<float>(nxt.tr[0]), 0.0f, 0.0f, 0.0f};
            float* loraA_sh = reinterpret_cast<float*>(smem_gen + oSmemLora) + ew * 4 * 32;  // this warp's [4][32]
            if (R0) {
            } else if (R1) {
                __syncwarp();  // the previous tile's reads are done
                loraA_sh[lane] = static_cast<float>(nxt.aval[0]);
                __syncwarp();
                fetch_fast(nxt_t, more, nxt);
            } else {
                tr[1] = static_cast<float>(nxt.tr[1]);
                tr[2] = static_cast<float>(nxt.tr[2]);
                tr[3] = static_cast<float>(nxt.tr[3]);
                __syncwarp();  // the previous tile's reads are done
#pragma unroll
                for (int r = 0; r < kTerms; ++r) loraA_sh[r * 32 + lane] = static_cast<float>(nxt.aval[r]);
                if constexpr (kStageNext) reinterpret_cast<int*>(next_sh)[lane] = nxt.next_b;
                __syncwarp();
                fetch_ctx(nxt_t, more, nxt);
            }

            // EPI_ADD_I8: this thread's 32 bytes of the residual stream, requested before the wait for the accumulator
            int4 res0 = make_int4(0, 0, 0, 0), res1 = make_int4(0, 0, 0, 0);
            bool res_vec = false;
            if constexpr (EPI == EPI_ADD_I8) {
                if (res_tma) {
                    have_cur = have_nxt;
                    rb_cur = rb_last;
                    issue_res_load(nxt_t, more);
                } else if (row_ok && chunk_ok) {
                    const int8_t* xr = p.resid + static_cast<size_t>(row) * p.ld_resid + col0;
                    res_vec = ((reinterpret_cast<uintptr_t>(xr) & 15) == 0) && (col0 + 32 <= p.n);
                    if (res_vec) {
                        res0 = *reinterpret_cast<const int4*>(xr);
                        res1 = *reinterpret_cast<const int4*>(xr + 16);
                    }
                }
            }

            // C, too, is requested before the wait (a 32 x 512 x 512 product added to another 5.4 -> 5.0 us; the instances with a rank term have no registers for it)
            constexpr bool kEarlyC = EPI == EPI_F32 && R0 && !PAIR && !B2;
            float4 c_early[kEarlyC ? 8 : 1];
            bool c_vec = false;
            if constexpr (kEarlyC) {
                if (p.beta != 0.0f && row_ok && col0 + 32 <= p.n) {
                    const float* crow = p.c + static_cast<size_t>(row) * p.ldc + col0;
                    c_vec = (reinterpret_cast<uintptr_t>(crow) & 15) == 0;
                    if (c_vec)
#pragma unroll
                        for (int j = 0; j < 8; ++j) c_early[j] = reinterpret_cast<const float4*>(crow)[j];
                }
            }

            ok = mbar_wait(bar_acc_full + 8 * buf, PAIR ? (pfull >> buf) & 1u : (it >> 1) & 1, 3);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            if constexpr (PAIR) pfull ^= 1u << buf;

            uint32_t acc[32];
            tmem_ld32(tmem_base + kAccCol + buf * BN + (static_cast<uint32_t>(q * 32) << 16) + c * 32, acc);
            tmem_ld_wait();
            // this warp no longer needs the accumulator: hand it back to the MMA warp
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if constexpr (PAIR) mbar_arrive_remote(acc_empty_bar + 8 * buf);
                else mbar_arrive(bar_acc_empty + 8 * buf);
            }
            if (!chunk_ok) continue;

            float v[32];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {  // packed fp32 pairs: each half rounds like the scalar instruction
                const float2 t2 = __fmul2_rn(make_float2(p.alpha, p.alpha), make_float2(__uint_as_float(acc[j]), __uint_as_float(acc[j + 1])));
                v[j] = t2.x;
                v[j + 1] = t2.y;
            }
            if (!R1 && p.beta != 0.0f && row_ok) {
                const float* crow = p.c + static_cast<size_t>(row) * p.ldc + col0;
                if (kEarlyC ? c_vec : col0 + 32 <= p.n && (reinterpret_cast<uintptr_t>(crow) & 15) == 0) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 c4 = kEarlyC ? c_early[kEarlyC ? j : 0] : reinterpret_cast<const float4*>(crow)[j];
                        v[4 * j] = fmaf(p.beta, c4.x, v[4 * j]);
                        v[4 * j + 1] = fmaf(p.beta, c4.y, v[4 * j + 1]);
                        v[4 * j + 2] = fmaf(p.beta, c4.z, v[4 * j + 2]);
                        v[4 * j + 3] = fmaf(p.beta, c4.w, v[4 * j + 3]);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (col0 + j < p.n) v[j] = fmaf(p.beta, crow[j], v[j]);
                }
            }
            const float lsign = (member & 1) ? -p.lora_scale : p.lora_scale;
            if constexpr (R1) {
                // t * A is an integer below 2^24: float products are exact
                const float2 tr2 = make_float2(tr[0], tr[0]), ls2 = make_float2(lsign, lsign);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 a4 = *reinterpret_cast<const float4*>(loraA_sh + 4 * j);
                    const float2 lo = __ffma2_rn(ls2, __fmul2_rn(tr2, make_float2(a4.x, a4.y)), make_float2(v[4 * j + 0], v[4 * j + 1]));
                    const float2 hi = __ffma2_rn(ls2, __fmul2_rn(tr2, make_float2(a4.z, a4.w)), make_float2(v[4 * j + 2], v[4 * j + 3]));
                    v[4 * j + 0] = lo.x; v[4 * j + 1] = lo.y; v[4 * j + 2] = hi.x; v[4 * j + 3] = hi.y;
                }
            } else if constexpr (!R0) {
                // sum_r t[r]*A[n][r] is an integer below 2^24: float products and sums are exact. Rows of another pair (and rows past m)
                // take part with a zero factor.
                const int pair_hi = kInside ? 0 : __shfl_sync(0xffffffffu, pair, 31);
                for (int pr = kInside ? 0 : __shfl_sync(0xffffffffu, pair, 0);; ++pr) {
                    const float ls = kInside || pair == pr ? lsign : 0.0f;
                    const float2 ls2 = make_float2(ls, ls);
                    const float2 t0 = make_float2(tr[0], tr[0]), t1 = make_float2(tr[1], tr[1]), t2 = make_float2(tr[2], tr[2]), t3 = make_float2(tr[3], tr[3]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 a0 = *reinterpret_cast<const float4*>(loraA_sh + 4 * j);
                        float2 lo = __fmul2_rn(t0, make_float2(a0.x, a0.y)), hi = __fmul2_rn(t0, make_float2(a0.z, a0.w));
                        auto add = [&](const float2 tt, int r) {
                            const float4 a = *reinterpret_cast<const float4*>(loraA_sh + 32 * r + 4 * j);
                            lo = __ffma2_rn(tt, make_float2(a.x, a.y), lo);
                            hi = __ffma2_rn(tt, make_float2(a.z, a.w), hi);
                        };
                        add(t1, 1);
                        if constexpr (kTerms > 2) { add(t2, 2); add(t3, 3); }
                        lo = __ffma2_rn(ls2, lo, make_float2(v[4 * j + 0], v[4 * j + 1]));
                        hi = __ffma2_rn(ls2, hi, make_float2(v[4 * j + 2], v[4 * j + 3]));
                        v[4 * j + 0] = lo.x; v[4 * j + 1] = lo.y; v[4 * j + 2] = hi.x; v[4 * j + 3] = hi.y;
                    }
                    if (kInside || pr >= pair_hi) break;
                    __syncwarp();  // the next pair's factor takes the place of this one's
                    int av[4] = {0, 0, 0, 0};
                    if (col0 + lane < p.n) load_a(pr + 1, col0 + lane, av);
#pragma unroll
                    for (int r = 0; r < kTerms; ++r) loraA_sh[r * 32 + lane] = static_cast<float>(av[r]);
                    __syncwarp();
                }
            }

            if constexpr (EPI == EPI_F32) {
                if (args.use_tma_store) {
                    // stage the 32x32 box in 128B-swizzled shared memory, then one TMA store (clips at M and N)
                    if (it > 0) {
                        if (lane == 0) bulk_wait_read<0>();
                        __syncwarp();
                    }
                    float4* dst = reinterpret_cast<float4*>(epi_gen + lane * 128);
#pragma unroll
                    for (int j = 0; j < 8; ++j) dst[j ^ (lane & 7)] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(&map_d, epi_buf, col0, m0 + q * 32);
                        bulk_commit();
                    }
                } else if (row_ok) {
                    float* drow = p.d + static_cast<size_t>(row) * p.ldd + col0;
                    const bool vec = ((reinterpret_cast<uintptr_t>(drow) & 15) == 0) && (col0 + 32 <= p.n);
                    if (vec) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) reinterpret_cast<float4*>(drow)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (col0 + j < p.n) drow[j] = v[j];
                    }
                }
            } else if constexpr (EPI == EPI_F16) {
                if (col0 < p.n_f16) {
                    // 32 rows x 32 halves staged as 64-byte rows, then one TMA store (clips at M; n_f16 is a multiple of 32).
                    // Two staging halves alternate, so only the store before the previous one has to have left shared memory.
                    if (lane == 0) bulk_wait_read<1>();
                    __syncwarp();
                    // 64B swizzle (16-byte piece ^ (row / 2) % 4): eight lanes' pieces fall into different banks. (Unswizzled, the stores' four-way conflicts
                    // took 59 % of the shared-memory wavefronts: 262144 x 1537 x 512 rank 1 215 -> 205 us, rank 4 336 -> 279.)
                    uint4* dst = reinterpret_cast<uint4*>(epi_gen + stage_half * 2048 + lane * 64);
                    const int sw = (lane >> 1) & 3;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const __half2 h0 = __floats2half2_rn(v[8 * j], v[8 * j + 1]), h1 = __floats2half2_rn(v[8 * j + 2], v[8 * j + 3]);
                        const __half2 h2 = __floats2half2_rn(v[8 * j + 4], v[8 * j + 5]), h3 = __floats2half2_rn(v[8 * j + 6], v[8 * j + 7]);
                        dst[j ^ sw] = make_uint4(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1),
                                                 *reinterpret_cast<const uint32_t*>(&h2), *reinterpret_cast<const uint32_t*>(&h3));
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_2d(&map_d, epi_buf + stage_half * 2048, col0, m0 + q * 32);
                        bulk_commit();
                    }
                    stage_half ^= 1;
                } else if (R1) {  // (the rank-1 instance runs with at most one fp32 column behind the halves)
                    if (col0 == p.n_f16) p.d[static_cast<size_t>(row) * p.ldd] = v[0];
                } else if (row_ok) {
                    float* drow = p.d + static_cast<size_t>(row) * p.ldd + (col0 - p.n_f16);
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (col0 + j < p.n) drow[j] = v[j];
                }
            } else if constexpr (EPI == EPI_ADD_I8) {
                if (res_tma) {
                    if (have_cur) {
                        ok = __all_sync(0xffffffffu, mbar_wait(rbar + 8 * rb_cur, (r_par >> rb_cur) & 1u, 5));
                        if (!ok) break;
                        r_par ^= 1u << rb_cur;
                        int4* rrow = reinterpret_cast<int4*>(epi_gen + rb_cur * 1024 + lane * 32);
                        const int sw = (lane >> 2) & 1;  // 32B swizzle: 16-byte piece ^ (row / 4) % 2
                        res0 = rrow[sw];
                        res1 = rrow[sw ^ 1];
                        const uint32_t rw[8] = {static_cast<uint32_t>(res0.x), static_cast<uint32_t>(res0.y), static_cast<uint32_t>(res0.z), static_cast<uint32_t>(res0.w),
                                                static_cast<uint32_t>(res1.x), static_cast<uint32_t>(res1.y), static_cast<uint32_t>(res1.z), static_cast<uint32_t>(res1.w)};
                        uint32_t upd[8];
#pragma unroll
                        for (int g = 0; g < 8; ++g) upd[g] = resid_add_word(rw[g], v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3], p.add_scale);
                        rrow[sw] = make_int4(static_cast<int>(upd[0]), static_cast<int>(upd[1]), static_cast<int>(upd[2]), static_cast<int>(upd[3]));
                        rrow[sw ^ 1] = make_int4(static_cast<int>(upd[4]), static_cast<int>(upd[5]), static_cast<int>(upd[6]), static_cast<int>(upd[7]));
                        fence_async_smem();
                        __syncwarp();
                        if (lane == 0) {  // clips at M and N
                            tma_store_2d(&map_d, epi_buf + rb_cur * 1024, col0, m0 + q * 32);
                            bulk_commit();
                        }
                    }
                } else if (row_ok) {
                    int8_t* xr = p.resid + static_cast<size_t>(row) * p.ld_resid + col0;
                    if (res_vec) {
                        const uint32_t rw[8] = {static_cast<uint32_t>(res0.x), static_cast<uint32_t>(res0.y), static_cast<uint32_t>(res0.z), static_cast<uint32_t>(res0.w),
                                                static_cast<uint32_t>(res1.x), static_cast<uint32_t>(res1.y), static_cast<uint32_t>(res1.z), static_cast<uint32_t>(res1.w)};
                        uint32_t upd[8];
#pragma unroll
                        for (int g = 0; g < 8; ++g) upd[g] = resid_add_word(rw[g], v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3], p.add_scale);
                        reinterpret_cast<int4*>(xr)[0] = make_int4(static_cast<int>(upd[0]), static_cast<int>(upd[1]), static_cast<int>(upd[2]), static_cast<int>(upd[3]));
                        reinterpret_cast<int4*>(xr)[1] = make_int4(static_cast<int>(upd[4]), static_cast<int>(upd[5]), static_cast<int>(upd[6]), static_cast<int>(upd[7]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            if (col0 + j < p.n) {
                                const float t = resid_add_biased(static_cast<float>(xr[j]), v[j], p.add_scale);
                                xr[j] = static_cast<int8_t>(__float_as_int(t) - kRoundBiasBits);
                            }
                        }
                    }
                }
            } else {
                // GELU -> int8 (reference: src/cuda_kernels.cu:3178-3194; tanh-form GELU, clip to +-127)
                if (!R1 && col0 + 32 > p.n) {  // (the rank-1 instance runs with n a multiple of 32)
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (col0 + j >= p.n) v[j] = 0.0f;  // gelu(0) = 0
                }
                // One 16-element scale block at a time: its 16 values take the fast evaluation in one straight-line stretch (no
                // branch between groups, so the scheduler interleaves them); a group with a value too close to a rounding
                // boundary is flagged and redone with the tanhf form (about one group in ten thousand), and a block that saturates is clamped. tb holds the
                // rounded values still biased by 1.5 * 2^23: the low byte of the bit pattern is the int8.
                // What bounds this: issue slots (about 20 per value, the special-function unit's 2.5 of them take it 65 % of the time). 262144 x 1024 x 512 rank 1 272 -> 249 us,
                // 65536 x 8192 x 2048 rank 4 943 -> 787, 4096 x 1024 x 512 without a rank term 9.9 -> 7.5, with the clamp and the |x| dependent tolerance
                // taken out of the common path and the codes' products unsnapped. One test per 8 or 16 values spills (254 -> 257, 264).
                // entry address from the bit pattern of (amax + kRoundBias): (bits - kRoundBiasBits) * 8, folded into one constant
                const uint32_t tab_c = smem_base + oSmemEpi - (static_cast<uint32_t>(kRoundBiasBits) << 3);
                const float safe = gelu_q8_safe(p.act_scale);
                int w[8];
                uint32_t sfv[2] = {0u, 0u}, codes[4] = {0u, 0u, 0u, 0u};
                int4 nb0 = make_int4(0, 0, 0, 0), nb1 = nb0;  // R1: the next projection's vector
#pragma unroll
                for (int blk = 0; blk < 2; ++blk) {
                    float tb[16];
                    float am = 0.0f;  // max |value| of the block
                    // (requested behind the second block's math: 262144 x 1024 x 512 277.9 us with the loads where they are used, 273 in front of both
                    // blocks, 281 in front of the accumulator wait, 271 here)
                    if constexpr (R1 && EPI == EPI_GELU_FP4) {
                        if (blk == 1) {
                            const int4* bv = reinterpret_cast<const int4*>(p.next_tvec + static_cast<size_t>(pair) * p.next_tvec_pair_stride + col0);
                            nb0 = __ldg(bv);
                            nb1 = __ldg(bv + 1);
                        }
                    }
                    float n16[16];  // R1: the integers as floats (the other instances have no registers for them: 250 instead of 201 us at 131072 x 1024 x 512 rank 4)
                    uint32_t bad = 0;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        float worst = 0.0f;
#pragma unroll
                        for (int e = 4 * g; e < 4 * g + 4; e += 2) {
                            float fc[2];
                            gelu_q8_fast2(v[16 * blk + e], v[16 * blk + e + 1], p.act_scale, worst, tb[e], tb[e + 1], fc[0], fc[1]);
                            am = fmax3(am, fabsf(fc[0]), fabsf(fc[1]));
                            n16[e] = fc[0];
                            n16[e + 1] = fc[1];
                        }
                        bad |= worst < safe ? 0u : (1u << g);
                    }
                    if (bad != 0) {
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            if ((bad >> g) & 1u) {
                                const int j = 16 * blk + 4 * g;
                                float tbx[4], fcx[4];
                                gelu_q8_exact4(v[j], v[j + 1], v[j + 2], v[j + 3], p.act_scale, tbx, fcx);
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    tb[4 * g + e] = tbx[e];
                                    n16[4 * g + e] = fcx[e];
                                }
                            }
                        }
                        am = 0.0f;
#pragma unroll
                        for (int e = 0; e < 16; ++e) am = fmaxf(am, fabsf(tb[e] - kRoundBias));
                    }
                    if (am > 127.0f) {
                        clamp_biased<16>(tb);
#pragma unroll
                        for (int e = 0; e < 16; ++e) n16[e] = tb[e] - kRoundBias;
                        am = 127.0f;
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g)
                        w[4 * blk + g] = static_cast<int>(__byte_perm(__byte_perm(__float_as_uint(tb[4 * g]), __float_as_uint(tb[4 * g + 1]), 0x0040),
                                                                      __byte_perm(__float_as_uint(tb[4 * g + 2]), __float_as_uint(tb[4 * g + 3]), 0x0040), 0x5410));
                    if constexpr (EPI == EPI_GELU_FP4) {
                        // {1 / scale, scale byte} of the block from the table; the codes from the conversion instruction
                        // applied to n / scale (e2m1x8_table)
                        uint32_t rbits, sbyte;
                        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(rbits), "=r"(sbyte) : "r"((__float_as_uint(am + kRoundBias) << 3) + tab_c));
                        sfv[blk] = sbyte;
                        codes[2 * blk] = R1 ? e2m1x8_table(n16, __uint_as_float(rbits)) : e2m1x8_biased(tb, __uint_as_float(rbits));
                        codes[2 * blk + 1] = R1 ? e2m1x8_table(n16 + 8, __uint_as_float(rbits)) : e2m1x8_biased(tb + 8, __uint_as_float(rbits));
                    }
                }
                if (!(R1 && EPI == EPI_GELU_FP4) && row_ok && p.d_i8 != nullptr) {  // (the rank-1 FP4 instance writes no int8 copy)
                    int8_t* drow = p.d_i8 + static_cast<size_t>(row) * p.ld_i8 + col0;
                    if (((reinterpret_cast<uintptr_t>(drow) & 15) == 0) && col0 + 32 <= p.n) {
                        reinterpret_cast<int4*>(drow)[0] = make_int4(w[0], w[1], w[2], w[3]);
                        reinterpret_cast<int4*>(drow)[1] = make_int4(w[4], w[5], w[6], w[7]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (col0 + j < p.n) drow[j] = static_cast<int8_t>((w[j >> 2] >> (8 * (j & 3))) & 0xff);
                    }
                }
                if constexpr (EPI == EPI_GELU_FP4) {
                    const bool one_pair = kInside || !kStageNext || __shfl_sync(0xffffffffu, pair, 0) == __shfl_sync(0xffffffffu, pair, 31);
                    if (row_ok) {
                        const uint32_t s0 = sfv[0], s1 = sfv[1], lo0 = codes[0], hi0 = codes[1], lo1 = codes[2], hi1 = codes[3];
                        *reinterpret_cast<uint4*>(p.d_codes + (static_cast<size_t>(row) * p.n + col0) / 2) = make_uint4(lo0, hi0, lo1, hi1);
                        const int kb = col0 >> 4;
                        *reinterpret_cast<uint16_t*>(p.d_sf + sf_offset(static_cast<int>(row), kb, sf_k_atoms(p.n))) =
                            static_cast<uint16_t>(s0 | (s1 << 8));
                        if ((!kStageNext || !one_pair) && (R1 || p.next_nvec > 0)) {  // (the rank-1 FP4 instance always feeds one projection)
                            const int8_t* tv = p.next_tvec + static_cast<size_t>(pair) * p.next_tvec_pair_stride + col0;
                            const int nv_ = R1 ? 1 : p.next_nvec;  // (the rank-1 instance runs with at most one projection)
                            for (int vv = 0; vv < nv_; ++vv) {
                                const int4* bv = reinterpret_cast<const int4*>(tv + static_cast<size_t>(vv) * p.n);
                                const int4 b0 = R1 ? nb0 : __ldg(bv), b1 = R1 ? nb1 : __ldg(bv + 1);
                                int a = 0;
                                a = __dp4a(w[0], b0.x, a); a = __dp4a(w[1], b0.y, a); a = __dp4a(w[2], b0.z, a); a = __dp4a(w[3], b0.w, a);
                                a = __dp4a(w[4], b1.x, a); a = __dp4a(w[5], b1.y, a); a = __dp4a(w[6], b1.z, a); a = __dp4a(w[7], b1.w, a);
                                atomicAdd(p.next_t + static_cast<size_t>(row) * p.next_nvec + vv, a);
                            }
                        }
                    }
                    if (kStageNext && one_pair) {  // (vectors that are not there are zeros; rows past m take part up to the store)
                        int a4[kTerms];
#pragma unroll
                        for (int vv = 0; vv < kTerms; ++vv) {
                            const int4 b0 = next_sh[2 * vv], b1 = next_sh[2 * vv + 1];
                            int a = 0;
                            a = __dp4a(w[0], b0.x, a); a = __dp4a(w[1], b0.y, a); a = __dp4a(w[2], b0.z, a); a = __dp4a(w[3], b0.w, a);
                            a = __dp4a(w[4], b1.x, a); a = __dp4a(w[5], b1.y, a); a = __dp4a(w[6], b1.z, a); a = __dp4a(w[7], b1.w, a);
                            a4[vv] = a;
                        }
                        if (p.next_nvec == kTerms) {
                            int* sums = reinterpret_cast<int*>(next_sh + 8);
                            if constexpr (kTerms == 2) reinterpret_cast<int2*>(sums)[lane] = make_int2(a4[0], a4[1]);
                            else reinterpret_cast<int4*>(sums)[lane] = make_int4(a4[0], a4[1], a4[kTerms - 2], a4[kTerms - 1]);
                            __syncwarp();
                            int* t = p.next_t + (static_cast<size_t>(m0) + q * 32) * kTerms + lane;
                            if (m0 + BM <= p.m) {
#pragma unroll
                                for (int i = 0; i < kTerms; ++i) atomicAdd(t + 32 * i, sums[32 * i + lane]);
                            } else {
                                for (int i = 0; i < kTerms; ++i)
                                    if (m0 + q * 32 + (32 * i + lane) / kTerms < p.m) atomicAdd(t + 32 * i, sums[32 * i + lane]);
                            }
                        } else if (row_ok) {
#pragma unroll
                            for (int vv = 0; vv < kTerms - 1; ++vv)
                                if (vv < p.next_nvec) atomicAdd(p.next_t + static_cast<size_t>(row) * p.next_nvec + vv, a4[vv]);
                        }
                    }
                }
            }
        }
        if constexpr (EPI == EPI_F32 || EPI == EPI_F16 || EPI == EPI_ADD_I8) {
            if (args.use_tma_store) {
                if (lane == 0) bulk_wait_read<0>();
                __syncwarp();
            }
        }
    }

    tc_fence_before();
    if constexpr (PAIR) cluster_sync();  // neither CTA leaves while the other may still signal or read it
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if constexpr (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols);
        else tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// Encoding a tensor map costs about half a microsecond of host time, as much as the rest of a launch's preparation, and callers
// keep their buffers: each thread keeps the maps of its last calls (direct-mapped, 256 entries, no device memory). A map is a
// pure function of its key.
struct MapKey {
    const void* base;
    uint64_t dim0, dim1, stride1, dim2, stride2;  // dim2 = 0: two dimensions
    uint32_t box0, box1, box2;
    int dt, swizzle;
    bool operator==(const MapKey& o) const {
        return base == o.base && dim0 == o.dim0 && dim1 == o.dim1 && stride1 == o.stride1 && dim2 == o.dim2 && stride2 == o.stride2 && box0 == o.box0 && box1 == o.box1 && box2 == o.box2 && dt == o.dt && swizzle == o.swizzle;
    }
};
struct MapSlot {
    MapKey key;
    CUtensorMap map;
};
constexpr unsigned kMapSlots = 256;

}  // namespace
int make_map_3d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t dim0, uint64_t dim1, uint64_t dim2, uint64_t stride1_bytes, uint64_t stride2_bytes,
                uint32_t box0, uint32_t box1, uint32_t box2, const char* what, CUtensorMapSwizzle swizzle) {
    static thread_local std::vector<MapSlot> cache;
    if (cache.empty()) cache.resize(kMapSlots, MapSlot{});
    const MapKey key{base, dim0, dim1, stride1_bytes, dim2, stride2_bytes, box0, box1, box2, static_cast<int>(dt), static_cast<int>(swizzle)};
    const uint64_t hash = mix_u64(reinterpret_cast<uint64_t>(base), mix_u64(dim0 ^ (static_cast<uint64_t>(box1) << 48), dim1 ^ (stride1_bytes << 24)));
    MapSlot& slot = cache[hash % kMapSlots];
    if (base != nullptr && slot.key == key) {
        *map = slot.map;
        return BNF4_OK;
    }
    EncodeTiledFn fn = get_encode_fn();
    if (fn == nullptr) return set_error(BNF4_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[3] = {dim0, dim1, dim2};
    const cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
    const cuuint32_t box[3] = {box0, box1, box2};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, dt, dim2 == 0 ? 2 : 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(BNF4_ERR_CUDA, "cuTensorMapEncodeTiled(%s) failed with %d", what, static_cast<int>(r));
    slot.key = key;
    slot.map = *map;
    return BNF4_OK;
}
int make_map_2d(CUtensorMap* map, CUtensorMapDataType dt, const void* base, uint64_t dim0, uint64_t dim1, uint64_t stride1_bytes,
                uint32_t box0, uint32_t box1, const char* what, CUtensorMapSwizzle swizzle) {
    return make_map_3d(map, dt, base, dim0, dim1, 0, stride1_bytes, 0, box0, box1, 1, what, swizzle);
}
namespace {

template <int EPI, int RK, bool PAIR, bool B2>
int launch_t(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& md, const ExtraMaps<PAIR, B2>& msf, const KernelArgs& args,
             dim3 grid, int dev, cudaStream_t stream) {
    constexpr int smem = PAIR ? kPairSmemAlloc : kSmemAlloc;
    static bool configured[64] = {};  // function attributes are per device: set once for each device this process uses
    if (!configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_nvfp4_kernel<EPI, RK, PAIR, B2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(gemm_nvfp4_kernel)");
        configured[dev] = true;
    }
    if constexpr (PAIR) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = kThreads;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, gemm_nvfp4_kernel<EPI, RK, PAIR, B2>, ma, mb, md, msf, args);
    } else {
        // (an early launch pays while the kernel is short: a dozen tiles per SM)
        launch_pdl_if(args.total_tiles <= 12 * static_cast<int>(grid.x), gemm_nvfp4_kernel<EPI, RK, PAIR, B2>, grid, kThreads, smem, stream, ma, mb, md, msf, args);
    }
    return check_launch("gemm_nvfp4_kernel");
}

}  // namespace

int gemm_nvfp4_launch(const GemmParams& p, cudaStream_t stream) {
    if (p.m <= 0 || p.n <= 0) return BNF4_OK;
    if (p.k <= 0 || (p.k % 64) != 0) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: k=%d must be a positive multiple of 64", p.k);
    if (!p.a || !p.b || !p.sfa || !p.sfb) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: null operand");
    if ((reinterpret_cast<uintptr_t>(p.a) & 15) || (reinterpret_cast<uintptr_t>(p.b) & 15) || (reinterpret_cast<uintptr_t>(p.sfa) & 15) ||
        (reinterpret_cast<uintptr_t>(p.sfb) & 15))
        return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: operands and scale factors must be 16-byte aligned");
    if (p.beta != 0.0f && p.c == nullptr) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: beta != 0 needs C");
    if (p.rank < 0 || p.rank > 4) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: rank=%d outside [0,4]", p.rank);
    if (p.rank > 0 && (!p.lora_t || !p.lora_A)) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: rank > 0 needs t and A");
    if (p.group_cols > 0 && (p.group_cols % 32) != 0) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: group_cols must be a multiple of 32");
    if (p.epilogue == EPI_F32 && !p.d) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: null D");
    if (p.epilogue == EPI_GELU_I8 && !p.d_i8) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: null int8 D");
    if (p.epilogue == EPI_ADD_I8 && (!p.resid || p.ld_resid < p.n)) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: the residual epilogue needs resid and ld_resid >= n");
    if (p.epilogue == EPI_F16) {
        if (!p.d_f16 || p.n_f16 <= 0 || (p.n_f16 % 32) != 0 || p.n_f16 > p.n) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: the fp16 epilogue needs d_f16 and n_f16 a multiple of 32 within n");
        if ((reinterpret_cast<uintptr_t>(p.d_f16) & 15) || (p.ld_f16 % 8) != 0 || p.ld_f16 < p.n_f16) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: fp16 D misaligned");
        if (p.n > p.n_f16 && (!p.d || p.ldd < p.n - p.n_f16)) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: the fp32 tail of the fp16 epilogue needs d and ldd >= n - n_f16");
    }
    if (p.epilogue == EPI_GELU_FP4) {
        if (!p.d_codes || !p.d_sf) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: null FP4 D");
        if ((p.n % 32) != 0) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: FP4 output needs n %% 32 == 0");
        if ((reinterpret_cast<uintptr_t>(p.d_codes) & 15) || (reinterpret_cast<uintptr_t>(p.d_sf) & 3))
            return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: FP4 output misaligned");
        if (p.next_nvec < 0 || p.next_nvec > 4) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: next_nvec outside [0,4]");
        if (p.next_nvec > 0 && ((reinterpret_cast<uintptr_t>(p.next_tvec) & 15) || (p.next_tvec_pair_stride & 15)))
            return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: next_tvec misaligned");
    }

    CUtensorMap ma, mb, md;
    int rc = make_map_2d(&ma, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.a, static_cast<uint64_t>(p.k) / 2, static_cast<uint64_t>(p.m),
                         static_cast<uint64_t>(p.k) / 2, 128, BM, "A");
    if (rc) return rc;
    rc = make_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.b, static_cast<uint64_t>(p.k) / 2, static_cast<uint64_t>(p.n),
                     static_cast<uint64_t>(p.k) / 2, 128, BN, "B");
    if (rc) return rc;
    KernelArgs args;
    args.p = p;
    args.k_atoms = sf_k_atoms(p.k);
    args.rpm_magic = p.rows_per_member > 0 ? static_cast<uint32_t>(std::min<unsigned long long>((1ull << 32) / static_cast<unsigned long long>(p.rows_per_member), 0xffffffffull)) : 0u;
    args.group_magic = p.group_cols > 0 ? static_cast<uint32_t>(((1ull << 32) + static_cast<unsigned long long>(p.group_cols) - 1) / static_cast<unsigned long long>(p.group_cols)) : 0u;
    if (p.group_cols > 0 && p.n >= 65536) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: column groups need n < 65536");
    args.lut = nullptr;
    if (p.epilogue == EPI_GELU_FP4) {
        args.lut = get_quant_lut();
        if (args.lut == nullptr) return BNF4_ERR_CUDA;
    }
    args.ks_wrap = p.b2 != nullptr ? (p.k + BK - 1) / BK : 0;
    args.use_tma_store = 0;
    if (p.epilogue == EPI_F32 && (reinterpret_cast<uintptr_t>(p.d) & 15) == 0 && (p.ldd % 4) == 0 && p.ldd >= p.n) {
        rc = make_map_2d(&md, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.d, static_cast<uint64_t>(p.n), static_cast<uint64_t>(p.m),
                         static_cast<uint64_t>(p.ldd) * 4, 32, 32, "D");
        if (rc) return rc;
        args.use_tma_store = g_gemm_allow_tma_store != 0;  // 0 direct stores, 1 TMA stores
    } else if (p.epilogue == EPI_F16) {
        // the half columns leave through a 32 x 32 box of halves (64-byte rows, 64B-swizzled staging)
        rc = make_map_2d(&md, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, p.d_f16, static_cast<uint64_t>(p.n_f16), static_cast<uint64_t>(p.m),
                         static_cast<uint64_t>(p.ld_f16) * 2, 32, 32, "D (fp16)", CU_TENSOR_MAP_SWIZZLE_64B);
        if (rc) return rc;
        args.use_tma_store = 1;
    } else if (p.epilogue == EPI_ADD_I8 && (reinterpret_cast<uintptr_t>(p.resid) & 15) == 0 && (p.ld_resid % 16) == 0) {
        // the residual stream enters and leaves through 32-row x 32-byte boxes
        rc = make_map_2d(&md, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.resid, static_cast<uint64_t>(p.n), static_cast<uint64_t>(p.m),
                         static_cast<uint64_t>(p.ld_resid), 32, 32, "residual stream", CU_TENSOR_MAP_SWIZZLE_32B);
        if (rc) return rc;
        args.use_tma_store = g_gemm_allow_tma_store != 0;
    } else {
        md = ma;  // unused
    }
    // (also called for the tiles of a pair)
    auto set_tiles = [&](int n_tiles, unsigned units) {
        args.n_tiles = n_tiles;
        args.tile_magic = n_tiles == 1 ? 0u : static_cast<uint32_t>(((1ull << 32) + static_cast<unsigned>(n_tiles) - 1) / static_cast<unsigned>(n_tiles));
        args.step_n = static_cast<int>(units % static_cast<unsigned>(n_tiles));
        args.step_m = static_cast<int>(units / static_cast<unsigned>(n_tiles));
    };
    args.n_tiles = (p.n + BN - 1) / BN;
    const long long tiles = static_cast<long long>(args.n_tiles) * ((p.m + BM - 1) / BM);
    if (tiles > 0x7fffffffLL) return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: too many tiles");
    args.total_tiles = static_cast<int>(tiles);
    int dev = 0;
    rc = current_device(&dev);
    if (rc) return rc;
    const int sms = multiprocessors(dev);
    if (sms <= 0) return BNF4_ERR_CUDA;
    const bool gelu = p.epilogue == EPI_GELU_FP4 || p.epilogue == EPI_GELU_I8;
    const bool gelu_plain = !gelu || ((p.n % 32) == 0 && (p.epilogue == EPI_GELU_FP4 ? (p.next_nvec == 1 && p.d_i8 == nullptr) : p.next_nvec <= 1));
    const bool plain = p.rank == 1 && p.beta == 0.0f && p.rows_per_member > 0 && (p.rows_per_member % BM) == 0 && (p.m % BM) == 0 && gelu_plain && (p.epilogue != EPI_F16 || p.n - p.n_f16 <= 1);
    const int rk = p.rank == 0 ? 0 : plain ? 1 : p.rank <= 2 && (p.epilogue != EPI_GELU_FP4 || p.next_nvec <= 2) ? 2 : 4;
    const int form = (p.rank == 2 || p.rank == 4) && rk == p.rank && (p.rows_per_member % 16) == 0 ? rk + 1 : rk;  // 32 rows lie in one pair
    // CTA pairs pay where the mainloop is longer than the epilogue. Measured at 65536 x 512, before the pairs' copies moved to their K steps (us, single
    // CTAs -> pairs): fp32 / half / residual epilogues, rank 1: K 512 33.9 -> 35.9, 25.6 -> 27.0, 29.0 -> 29.8; K 1024 42.7 -> 38.2,
    // 33.1 -> 30.2, 36.1 -> 33.1; K 4096 107 -> 80, 96 -> 70, 98 -> 74. Rank 4 with the last two: K 1024 37.2 -> 39.2, 43.3 -> 45.4, K 1536
    // 46.8 -> 43.3, 49.5 -> 47.4. GELU epilogues, whose math takes as long as K 1536: K 1536 52.7 -> 54.6, K 2048 63.8 -> 59.9, K 4096 105 -> 82.
    const long long pair_tiles = static_cast<long long>((p.n + 255) / 256) * ((p.m + 255) / 256);
    const int pair_k = gelu ? 2048 : (p.rank > 1 && p.epilogue != EPI_F32 ? 1536 : 1024);
    // Those are figures of many waves. In a few, whole waves of the larger tiles and the drain of their two epilogues decide: 10218 x 384 x 2240 took
    // 15.1 us with single CTAs and 25.0 with pairs, 7668 x 576 x 2880 21.7 and 26.6. So the two are compared by what they cost in waves, in us: K blocks of 256
    // at 0.44 and 0.6, epilogues of a sub-tile at 1.3 (GELU 1.9; 60 % more with the longer rank terms), 3 for starting a pair. Over 330 shapes of 0.5
    // to 16 k rows, 64 to 4096 columns and K 1024 to 4096 the choice costs 0.3 % on average against the better of the two and 16 % at most (GELU at K 1984, where
    // pairs pay by now; single CTAs throughout 2.4 %, pairs 37 %).
    auto waves_us = [&](long long t, int slots, float block, float epi) {
        const float nk = block * static_cast<float>((p.k + BK - 1) / BK);
        return nk + static_cast<float>((t + slots - 1) / slots - 1) * std::max(nk, epi) + epi;
    };
    const float epi_us = (gelu ? 1.9f : 1.3f) * (rk >= 2 ? 1.6f : 1.0f);
    const bool pair = p.b2 == nullptr && p.k >= pair_k && (rk != 1 || (p.m % 256) == 0) &&
                      3.0f + waves_us(pair_tiles, std::max(1, sms / 2), 0.6f, 2.0f * epi_us) < waves_us(tiles, sms, 0.44f, epi_us);
    // the epilogue and the form of the rank term are template arguments
    auto with_rank = [&](auto run) -> int {
        switch (form) {
            case 0: return run(std::integral_constant<int, 0>());
            case 1: return run(std::integral_constant<int, 1>());
            case 2: return run(std::integral_constant<int, 2>());
            case 3: return run(std::integral_constant<int, 3>());
            case 4: return run(std::integral_constant<int, 4>());
        }
        return run(std::integral_constant<int, 5>());
    };
    auto with_epilogue = [&](auto run) -> int {
        switch (p.epilogue) {
            case EPI_F32: return run(std::integral_constant<int, EPI_F32>());
            case EPI_GELU_I8: return run(std::integral_constant<int, EPI_GELU_I8>());
            case EPI_GELU_FP4: return run(std::integral_constant<int, EPI_GELU_FP4>());
            case EPI_ADD_I8: return run(std::integral_constant<int, EPI_ADD_I8>());
            case EPI_F16: return run(std::integral_constant<int, EPI_F16>());
        }
        return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: unknown epilogue %d", p.epilogue);
    };
    if (pair) {
        PairMaps msf;
        rc = make_map_2d(&mb, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.b, static_cast<uint64_t>(p.k) / 2, static_cast<uint64_t>(p.n), static_cast<uint64_t>(p.k) / 2, 128, 64, "B (pair)");
        if (!rc) rc = make_map_2d(&msf.sfa, CU_TENSOR_MAP_DATA_TYPE_UINT32, p.sfa, 128, static_cast<uint64_t>((p.m + 127) / 128) * args.k_atoms, 512, 128, 4, "A scales", CU_TENSOR_MAP_SWIZZLE_NONE);
        if (!rc) rc = make_map_2d(&msf.sfb, CU_TENSOR_MAP_DATA_TYPE_UINT32, p.sfb, 128, static_cast<uint64_t>((p.n + 127) / 128) * args.k_atoms, 512, 128, 4, "B scales", CU_TENSOR_MAP_SWIZZLE_NONE);
        if (rc) return rc;
        args.total_tiles = static_cast<int>(pair_tiles);
        const dim3 grid(2 * static_cast<unsigned>(std::min<long long>(pair_tiles, sms / 2)), 1, 1);
        set_tiles((p.n + 255) / 256, grid.x / 2);
        return with_epilogue([&](auto epi) -> int {
            constexpr int E = decltype(epi)::value;
            auto run = [&](auto r) { return launch_t<E, decltype(r)::value, true, false>(ma, mb, md, msf, args, grid, dev, stream); };
            return with_rank(run);
        });
    }
    if (gemm_panel_applies(p, rk, sms)) return gemm_panel_launch(p, rk, ma, mb, md, args.group_magic, sms, dev, stream);
    const dim3 grid(static_cast<unsigned>(std::min<long long>(tiles, sms)), 1, 1);
    set_tiles(args.n_tiles, grid.x);
    if (p.b2 != nullptr) {
        if (p.sfb2 == nullptr || (p.b2_rows % 128) != 0 || p.b2_rows < p.n || p.rows_per_member <= 0 || (p.rows_per_member % BM) != 0 || p.rank > 0)
            return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: the second operand needs member rows and b2_rows in multiples of 128 and takes no rank term");
        B2Map b2;
        const uint64_t members = (static_cast<uint64_t>(p.m) + p.rows_per_member - 1) / p.rows_per_member;
        rc = make_map_2d(&b2.b2, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.b2, static_cast<uint64_t>(p.k) / 2, members * p.b2_rows, static_cast<uint64_t>(p.k) / 2, 128, BN, "B2");
        if (rc) return rc;
        switch (p.epilogue) {  // (the dense form's)
            case EPI_F32: return launch_t<EPI_F32, 0, false, true>(ma, mb, md, b2, args, grid, dev, stream);
            case EPI_GELU_FP4: return launch_t<EPI_GELU_FP4, 0, false, true>(ma, mb, md, b2, args, grid, dev, stream);
            case EPI_ADD_I8: return launch_t<EPI_ADD_I8, 0, false, true>(ma, mb, md, b2, args, grid, dev, stream);
        }
        return set_error(BNF4_ERR_INVALID, "gemm_nvfp4: no second operand with epilogue %d", p.epilogue);
    }
    return with_epilogue([&](auto epi) -> int {
        constexpr int E = decltype(epi)::value;
        auto run = [&](auto r) { return launch_t<E, decltype(r)::value, false, false>(ma, mb, md, NoMaps{}, args, grid, dev, stream); };
        return with_rank(run);
    });
}

int gemm_nvfp4_device_error(cudaStream_t stream, int* out_code) {
    int rc = check_cuda(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
    if (rc) return rc;
    int code = 0;
    for (auto take : {take_wait_error, gemm_panel_device_error, efla_tc_device_error, efla_seq_device_error}) {
        int one = 0;
        rc = take(&one);
        if (rc) return rc;
        if (code == 0) code = one;
    }
    if (out_code) *out_code = code;
    if (code != 0) return set_error(BNF4_ERR_DEVICE, "a bounded wait expired in a kernel (code %d: up to 9 block-scaled GEMM, 11 to 20 scan on halves, 21 to 29 scan of wide heads, 31 to 39 panel GEMM)", code);
    return BNF4_OK;
}

}  // namespace bnf4
