// The block-scaled FP4 GEMM of gemm_tcgen05.cu with half outputs, for short contractions (K <= 512) and many rows: a CTA keeps one panel of B.
//
// With K this short a tile's product takes less time than its epilogue, and much of what the general kernel does per 128 x 128 tile does not depend on
// the tile: it fetches B and its scales again (72 of 108 KB), copies those scales to tensor memory (half of the scale copies), and its epilogue
// keeps books on members, groups and the pair's factor (100 of 258 instructions per warp). Here a CTA owns 256 columns: their B rows
// stay in shared memory, their scales in tensor memory, and it walks down the rows of A. The epilogue's per-tile state advances by constants
// and is fetched once for 256 columns; the factor of a pair is read when the pair changes. 262144 x 1537 x 512: no rank term 195 -> 173 us, rank 1
// 212 -> 180 (4.5 TB/s of output). It does not pay for the other epilogues: fp32 boxes leave one staging buffer per warp, which two
// passes of a tile then wait for (262144 x 256 64 -> 70 us), the GELU is bound by its own instructions (the same time), and higher ranks need more registers than
// are left (rank 2 297 -> 418 us, rank 4 267 -> 283).
//
// The CTAs of one panel take every `per`-th row tile, so that at any time all panels work on the same rows of A and read them from L2.
//
// Structure of one CTA (576 threads), as in the general kernel: warp 0 loads (the panel once, then A tiles of 128 rows x 256 K-elements into a
// ring of four), warp 1 issues scale copies and MMAs (M 128, N up to 256), warps 2..17 are the epilogue. Tensor memory holds three accumulator
// blocks of 128 columns: even tiles fill the first two, odd ones the last two, and the epilogue drains the shared block first, so that the next
// tile's product runs under the rest of the present epilogue. A panel of at most 128 columns alternates between the first two blocks.
// A single column behind the last whole panel (the stacked q | k | v | beta projection has 3 H + 1) is a second MMA of 16 columns per K step in
// that panel's CTAs, not a panel of its own.

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "tcgen05.cuh"

namespace bnf4 {

namespace {

constexpr int BM = 128, kWidth = 256;  // rows of a tile, columns of a panel
constexpr int BK = 256;       // K elements per stage (128 bytes of packed e2m1 per row)
constexpr int kMaxK = 512;
constexpr int kStages = 4;
constexpr int kStageABytes = BM * 128;
constexpr int kStageSfBytes = 4 * 512;
constexpr int kHalfBytes = 128 * 128;  // 128 rows of B, one K block
constexpr int kTailRows = 16;
constexpr int kTailBytes = kTailRows * 128;
constexpr int kEpiWarps = 16;
constexpr int kEpiBufBytes = 2 * 32 * 32 * 2;  // two boxes of 32 x 32 halves
constexpr int kThreads = 64 + kEpiWarps * 32;
constexpr int kEarlyTiles = 6;  // row tiles per CTA up to which an early launch pays

constexpr int kSmemA = 0;
constexpr int kSmemB = kSmemA + kStages * kStageABytes;        // [K block][half] of 128 rows
constexpr int kSmemTail = kSmemB + 4 * kHalfBytes;             // [K block]
constexpr int kSmemSfa = kSmemTail + 2 * kTailBytes;
constexpr int kSmemEpi = kSmemSfa + kStages * kStageSfBytes;
constexpr int kSmemLora = kSmemEpi + kEpiWarps * kEpiBufBytes;  // per epilogue warp: 64 floats of the pair's factor
constexpr int kSmemBar = kSmemLora + kEpiWarps * 64 * 4;
constexpr int kSmemAlloc = kSmemBar + 256 + 1024;
static_assert(kSmemAlloc <= 232448, "shared memory of one SM");
constexpr int kSmemSfb = kSmemA + (kStages - 1) * kStageABytes;  // the panel's scale atoms, in the last stage until they are in tensor memory
static_assert(3 * 8 * 512 <= kStageABytes, "scale atoms of both halves and the tail");

// tensor memory columns
constexpr int kTmemCols = 512;
constexpr int kSfbCol = 384;              // 8 per K step
constexpr int kSfaCol = kSfbCol + 64;     // 16: the pipe executes copies and MMAs in order, one slot suffices
constexpr int kTailCol = kSfaCol + 16;    // accumulator of the tail
constexpr int kTailSfCol = kTailCol + 16;  // 4 per K step
static_assert(kTailSfCol + 32 <= kTmemCols, "tensor memory");

constexpr uint32_t kIdescM128 = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(BM >> 4) << 24);  // see gemm_tcgen05.cu; N >> 3 at bit 17

struct PanelArgs {
    GemmParams p;
    int k_atoms;
    uint32_t group_magic;  // ceil(2^32 / group_cols) (0 when group_cols == 0)
    int m_tiles;
    int panels;  // blockIdx.x % panels is the CTA's panel
    int per;     // CTAs per panel: it takes row tiles blockIdx.x / panels + i * per
    int tail;    // 1: column n - 1, the only fp32 one, belongs to the last panel's CTAs
};

__device__ __forceinline__ void tmem_ld1(uint32_t taddr, uint32_t& r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
}

// RK as in the general kernel: 0 no rank term; 1 rank 1, members of whole row tiles, m a multiple of them, at most one fp32 column.
template <int RK>
__global__ void __launch_bounds__(kThreads, 1) gemm_panel_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                                                                 const __grid_constant__ CUtensorMap map_bt, const __grid_constant__ CUtensorMap map_d,
                                                                 const PanelArgs args) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

    const GemmParams& p = args.p;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int num_ks = (p.k + BK - 1) / BK;

    const uint32_t bar_full = smem_base + kSmemBar;          // kStages x 8 bytes
    const uint32_t bar_empty = bar_full + 8 * kStages;       // kStages
    const uint32_t bar_tile = bar_empty + 8 * kStages;       // 2: products of an even / odd tile complete
    const uint32_t bar_acc_empty = bar_tile + 16;            // 3 accumulator blocks
    const uint32_t bar_tail_empty = bar_acc_empty + 24;
    const uint32_t bar_panel = bar_tail_empty + 8;           // the panel has arrived
    const uint32_t bar_sfb = bar_panel + 8;                  // its scales are in tensor memory
    const uint32_t tmem_slot = bar_sfb + 8;
    volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + kSmemBar + (tmem_slot - bar_full));

    const int panel = static_cast<int>(blockIdx.x) % args.panels, mt0 = static_cast<int>(blockIdx.x) / args.panels;
    const int n0 = panel * kWidth;
    const bool tail = args.tail != 0 && panel == args.panels - 1;
    const int n_main = p.n - args.tail;                     // columns in whole panels
    const int width = min(kWidth, n_main - n0);
    const bool two = width > 128;                            // the panel fills a second block

    if (threadIdx.x == 64) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_b)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_d)) : "memory");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_tile, 1);
        mbar_init(bar_tile + 8, 1);
        for (int b = 0; b < 3; ++b) mbar_init(bar_acc_empty + 8 * b, kEpiWarps);
        mbar_init(bar_tail_empty, 4);
        mbar_init(bar_panel, 1);
        mbar_init(bar_sfb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot_gen;
    pdl_wait();

    if (warp == 0) {
        // ------------------------------ producer ------------------------------
        const uint32_t atoms_bytes = static_cast<uint32_t>(args.k_atoms) * 512u;
        if (elect_one()) {
            const int halves = two ? 2 : 1;
            mbar_expect_tx(bar_panel, static_cast<uint32_t>(halves * num_ks) * kHalfBytes + static_cast<uint32_t>(halves) * atoms_bytes +
                                          (tail ? static_cast<uint32_t>(num_ks) * kTailBytes + atoms_bytes : 0u));
            const uint8_t* sfb = static_cast<const uint8_t*>(p.sfb);
            for (int h = 0; h < halves; ++h) {
                for (int ks = 0; ks < num_ks; ++ks) tma_load_2d(smem_base + kSmemB + (2 * ks + h) * kHalfBytes, &map_b, ks * 128, n0 + 128 * h, bar_panel);
                bulk_load_1d(smem_base + kSmemSfb + h * 4096, sfb + static_cast<size_t>((n0 >> 7) + h) * atoms_bytes, atoms_bytes, bar_panel);
            }
            if (tail) {
                for (int ks = 0; ks < num_ks; ++ks) tma_load_2d(smem_base + kSmemTail + ks * kTailBytes, &map_bt, ks * 128, p.n - 1, bar_panel);
                bulk_load_1d(smem_base + kSmemSfb + 2 * 4096, sfb + static_cast<size_t>((p.n - 1) >> 7) * atoms_bytes, atoms_bytes, bar_panel);
            }
        }
        __syncwarp();
        int kc = 0, s = 0;
        uint32_t empty_parity = 1;
        bool ok = true;
        const uint8_t* sfa_src = static_cast<const uint8_t*>(p.sfa) + static_cast<size_t>(mt0) * atoms_bytes;
        const size_t sfa_step = static_cast<size_t>(args.per) * atoms_bytes;
        for (int mt = mt0; mt < args.m_tiles && ok; mt += args.per, sfa_src += sfa_step) {
            int atoms_left = args.k_atoms;
            for (int ks = 0; ks < num_ks; ++ks, ++kc) {
                if (kc >= kStages) ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, empty_parity, 31));
                else if (kc == kStages - 1) ok = __all_sync(0xffffffffu, mbar_wait(bar_sfb, 0, 36));  // the panel's scales have left this stage
                if (!ok) break;
                const uint32_t sf_bytes = static_cast<uint32_t>(min(4, atoms_left)) * 512u;
                atoms_left -= 4;
                const uint32_t bar = bar_full + 8 * s;
                if (elect_one()) {
                    mbar_expect_tx(bar, kStageABytes + sf_bytes);
                    tma_load_2d(smem_base + kSmemA + s * kStageABytes, &map_a, ks * 128, mt * BM, bar);
                    bulk_load_1d(smem_base + kSmemSfa + s * kStageSfBytes, sfa_src + ks * 2048, sf_bytes, bar);
                }
                __syncwarp();
                if (++s == kStages) { s = 0; empty_parity ^= 1u; }
            }
        }
        pdl_trigger();
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        const uint64_t adesc0 = smem_desc(smem_base + kSmemA, 16, 1024, kLayoutSw128);
        const uint64_t bdesc0 = smem_desc(smem_base + kSmemB, 16, 1024, kLayoutSw128);
        const uint64_t tdesc0 = smem_desc(smem_base + kSmemTail, 16, 1024, kLayoutSw128);
        const uint64_t sfadesc0 = smem_desc(smem_base + kSmemSfa, 0, 128, kLayoutNone);
        const uint64_t sfbdesc0 = smem_desc(smem_base + kSmemSfb, 0, 128, kLayoutNone);
        const uint32_t idesc = kIdescM128 | (static_cast<uint32_t>((width + 15) / 16 * 2) << 17);
        constexpr uint32_t idesc_tail = kIdescM128 | (static_cast<uint32_t>(kTailRows >> 3) << 17);
        bool ok = __all_sync(0xffffffffu, mbar_wait(bar_panel, 0, 32));
        tc_fence_after();
        if (ok && elect_one()) {
            for (int j = 0; j < args.k_atoms; ++j) {
                tc_cp_sf(tmem_base + kSfbCol + 8 * j, sfbdesc0 + static_cast<uint64_t>(j * (512 >> 4)));
                if (two) tc_cp_sf(tmem_base + kSfbCol + 8 * j + 4, sfbdesc0 + static_cast<uint64_t>((4096 + j * 512) >> 4));
                if (tail) tc_cp_sf(tmem_base + kTailSfCol + 4 * j, sfbdesc0 + static_cast<uint64_t>((8192 + j * 512) >> 4));
            }
            tc_commit(bar_sfb);
        }
        __syncwarp();
        int s = 0;
        uint32_t full_parity = 0, odd = 0, used = 0, empty_par = 0, tail_par = 1;
        for (int mt = mt0; mt < args.m_tiles && ok; mt += args.per, odd ^= 1u) {
            for (uint32_t b = odd; b <= odd + (two ? 1u : 0u) && ok; ++b) {  // the epilogue has drained the blocks
                if ((used >> b) & 1u) {
                    ok = __all_sync(0xffffffffu, mbar_wait(bar_acc_empty + 8 * b, (empty_par >> b) & 1u, 34));
                    empty_par ^= 1u << b;
                }
                used |= 1u << b;
            }
            if (tail && ok) {
                ok = __all_sync(0xffffffffu, mbar_wait(bar_tail_empty, tail_par, 35));  // (parity 1 first: passes at once)
                tail_par ^= 1u;
            }
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem_base + odd * 128;
            for (int ks = 0; ks < num_ks; ++ks) {
                ok = __all_sync(0xffffffffu, mbar_wait(bar_full + 8 * s, full_parity, 37));
                if (!ok) break;
                tc_fence_after();
                const int nk = min(4, args.k_atoms - 4 * ks);
                const uint64_t sfa_d = sfadesc0 + static_cast<uint64_t>(s * (kStageSfBytes >> 4));
                const uint64_t a_d = adesc0 + static_cast<uint64_t>(s * (kStageABytes >> 4));
                const uint64_t b_d = bdesc0 + static_cast<uint64_t>(ks * (2 * kHalfBytes >> 4));
                const uint64_t t_d = tdesc0 + static_cast<uint64_t>(ks * (kTailBytes >> 4));
                const uint32_t t_sfa = tmem_base + kSfaCol, t_sfb = tmem_base + kSfbCol + 32 * ks, t_sft = tmem_base + kTailSfCol + 16 * ks;
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j < nk) {
                            tc_cp_sf(t_sfa + 4 * j, sfa_d + static_cast<uint64_t>(j * (512 >> 4)));
                            tc_mma_nvf4(acc, a_d + static_cast<uint64_t>(j * (32 >> 4)), b_d + static_cast<uint64_t>(j * (32 >> 4)), idesc, t_sfa + 4 * j, t_sfb + 8 * j, ks > 0 || j > 0 ? 1u : 0u);
                        }
                    if (tail) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (j < nk) tc_mma_nvf4(tmem_base + kTailCol, a_d + static_cast<uint64_t>(j * (32 >> 4)), t_d + static_cast<uint64_t>(j * (32 >> 4)), idesc_tail, t_sfa + 4 * j, t_sft + 4 * j, ks > 0 || j > 0 ? 1u : 0u);
                    }
                    tc_commit(bar_empty + 8 * s);
                    if (ks == num_ks - 1) tc_commit(bar_tile + 8 * odd);
                }
                __syncwarp();
                if (++s == kStages) { s = 0; full_parity ^= 1u; }
            }
        }
    } else {
        // ------------------------------ epilogue: 16 warps, four per TMEM lane quadrant, 32 columns of each half ------------------------------
        constexpr bool R1 = RK == 1, R0 = RK == 0;
        const int ew = warp - 2;
        const int q = warp & 3;
        const int c = ew >> 2;
        const uint32_t epi_buf = smem_base + kSmemEpi + ew * kEpiBufBytes;
        uint8_t* epi_gen = smem_gen + kSmemEpi + ew * kEpiBufBytes;
        float* la = reinterpret_cast<float*>(smem_gen + kSmemLora) + ew * 64;  // this warp's [half][32]
        const int row_in_tile = q * 32 + lane;
        const int colh[2] = {n0 + c * 32, n0 + 128 + c * 32};  // first column of the warp's chunk in each half
        const bool chunk0 = colh[0] < n0 + width, chunk1 = colh[1] < n0 + width;
        const int z = static_cast<int>(opaque_zero());  // (read-only loads: their addresses depend on this)
        // projections: the group of a chunk is the CTA's for good
        auto group_of = [&](int col) { return p.group_cols > 0 ? static_cast<int>(__umulhi(static_cast<uint32_t>(col), args.group_magic)) : 0; };
        const int g0 = R0 ? 0 : group_of(min(colh[0], p.n - 1)) + z, g1 = R0 ? 0 : group_of(min(colh[1], p.n - 1)) + z;  // (chunks behind the last column have none of their own)
        const bool two_groups = !R0 && two && g0 != g1;
        const bool tail_warp = tail && c == 0;
        const int g_tail = R0 || !tail_warp ? 0 : group_of(p.n - 1) + z;
        // the next tile's projections (both halves' and the tail column's) are requested one tile ahead
        int nt0 = 0, nt1 = 0, ntt = 0;
        auto fetch_t = [&](int mt) {
            if (R0 || mt >= args.m_tiles) return;
            const int* t_ptr = p.lora_t + static_cast<size_t>(static_cast<unsigned>(mt * BM + row_in_tile)) * p.t_stride;
            nt0 = t_ptr[g0];
            if (two_groups) nt1 = t_ptr[g1];
            if (tail_warp) ntt = t_ptr[g_tail];
        };
        // member of the tile's rows; the warp's factor copy holds that of pair `held`
        int member = z, held = -1;
        int trk_member = z;
        long long trk_end = p.rows_per_member;
        auto element = [&](int pr, int col) { return __ldg(p.lora_A + static_cast<size_t>(pr) * p.lora_A_pair_stride + col); };
        int av0 = 0, av1 = 0, atail = 0;  // the next tile's pair, if it is another one
        auto fetch_a = [&](int pr) {
            if (colh[0] + lane < n_main) av0 = element(pr, colh[0] + lane);
            if (two && colh[1] + lane < n_main) av1 = element(pr, colh[1] + lane);
            if (tail_warp) atail = element(pr, p.n - 1);
        };
        auto hold_a = [&](int pr) {
            __syncwarp();  // earlier reads of the copy are done
            la[lane] = static_cast<float>(av0);
            la[32 + lane] = static_cast<float>(av1);
            __syncwarp();
            held = pr;
        };
        // tracks the members of whole row tiles by comparison
        auto track = [&](int mt) {
            while (static_cast<long long>(mt) * BM >= trk_end) { ++trk_member; trk_end += p.rows_per_member; }
        };
        int want = -1;  // the pair that av0 / av1 hold for the next tile (its first in this warp)
        fetch_t(mt0);
        if constexpr (R1) {
            track(mt0);
            want = trk_member >> 1;
            fetch_a(want);
        }
        int stage_half = 0;
        bool ok = true;
        uint32_t odd = 0, tile_par = 0;  // bit b: parity to wait for on bar_tile[b]
        unsigned row = static_cast<unsigned>(mt0 * BM + row_in_tile);  // (rows fit 31 bits)
        for (int mt = mt0; mt < args.m_tiles && ok; mt += args.per, row += static_cast<unsigned>(args.per * BM), odd ^= 1u) {
            const bool row_ok = R1 || row < static_cast<unsigned>(p.m);
            float t0 = 0.0f, t1 = 0.0f, tt = 0.0f;
            if constexpr (R1) {
                member = trk_member;
                if (want != held) hold_a(want);
                t0 = static_cast<float>(nt0);
                t1 = two_groups ? static_cast<float>(nt1) : t0;
                tt = static_cast<float>(ntt) * static_cast<float>(atail);
                fetch_t(mt + args.per);
                if (mt + args.per < args.m_tiles) {
                    track(mt + args.per);
                    if ((trk_member >> 1) != want) {
                        want = trk_member >> 1;
                        fetch_a(want);
                    }
                }
            }
            const float lsign = (member & 1) ? -p.lora_scale : p.lora_scale;

            ok = __all_sync(0xffffffffu, mbar_wait(bar_tile + 8 * odd, (tile_par >> odd) & 1u, 33));
            if (!ok) break;
            tile_par ^= 1u << odd;
            tc_fence_after();

            if (tail_warp) {
                uint32_t a;
                tmem_ld1(tmem_base + kTailCol + (static_cast<uint32_t>(q * 32) << 16), a);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_tail_empty);
                float v = __fmul_rn(p.alpha, __uint_as_float(a));
                if constexpr (R1) v = fmaf(lsign, tt, v);
                if (row_ok) p.d[static_cast<size_t>(row) * p.ldd] = v;
            }

#pragma unroll 1
            for (uint32_t pass = 0; pass < (two ? 2u : 1u); ++pass) {
                const uint32_t h = two ? pass ^ odd ^ 1u : 0u;  // the half in the shared block first
                const int col0 = h ? colh[1] : colh[0];
                const bool chunk_ok = h ? chunk1 : chunk0;
                uint32_t acc[32];
                tmem_ld32(tmem_base + (odd + h) * 128 + (static_cast<uint32_t>(q * 32) << 16) + c * 32, acc);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acc_empty + 8 * (odd + h));
                if (!chunk_ok) continue;

                float v[32];
#pragma unroll
                for (int j = 0; j < 32; j += 2) {  // packed fp32 pairs: each half rounds like the scalar instruction
                    const float2 t2 = __fmul2_rn(make_float2(p.alpha, p.alpha), make_float2(__uint_as_float(acc[j]), __uint_as_float(acc[j + 1])));
                    v[j] = t2.x;
                    v[j + 1] = t2.y;
                }
                const float* lh = la + h * 32;
                if constexpr (R1) {
                    // t * A is an integer below 2^24: float products are exact
                    const float t = h ? t1 : t0;
                    const float2 tr2 = make_float2(t, t), ls2 = make_float2(lsign, lsign);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 a4 = *reinterpret_cast<const float4*>(lh + 4 * j);
                        const float2 lo = __ffma2_rn(ls2, __fmul2_rn(tr2, make_float2(a4.x, a4.y)), make_float2(v[4 * j + 0], v[4 * j + 1]));
                        const float2 hi = __ffma2_rn(ls2, __fmul2_rn(tr2, make_float2(a4.z, a4.w)), make_float2(v[4 * j + 2], v[4 * j + 3]));
                        v[4 * j + 0] = lo.x; v[4 * j + 1] = lo.y; v[4 * j + 2] = hi.x; v[4 * j + 3] = hi.y;
                    }
                }

                if (col0 < p.n_f16) {
                    // 32 rows x 32 halves staged as 64-byte rows (64B swizzle), then one TMA store; two staging halves alternate
                    if (lane == 0) bulk_wait_read<1>();
                    __syncwarp();
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
                        tma_store_2d(&map_d, epi_buf + stage_half * 2048, col0, mt * BM + q * 32);
                        bulk_commit();
                    }
                    stage_half ^= 1;
                } else if (row_ok) {
                    float* drow = p.d + static_cast<size_t>(row) * p.ldd + (col0 - p.n_f16);
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (col0 + j < n_main) drow[j] = v[j];
                }
            }
        }
        if (lane == 0) bulk_wait_read<0>();
        __syncwarp();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

template <int RK>
int launch_t(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mbt, const CUtensorMap& md, const PanelArgs& args, int dev, cudaStream_t stream) {
    static bool configured[64] = {};
    if (!configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_panel_kernel<RK>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemAlloc);
        if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(gemm_panel_kernel)");
        configured[dev] = true;
    }
    // (an early launch pays while the kernel is short)
    launch_pdl_if(args.m_tiles <= kEarlyTiles * args.per, gemm_panel_kernel<RK>, dim3(static_cast<unsigned>(args.panels * args.per)), kThreads, kSmemAlloc, stream, ma, mb, mbt, md, args);
    return check_launch("gemm_panel_kernel");
}

// One fp32 column behind whole panels is no panel of its own.
int tail_column(const GemmParams& p) { return p.n > kWidth && p.n % kWidth == 1 && p.n_f16 == p.n - 1 ? 1 : 0; }
int panels_of(const GemmParams& p) { return (p.n - tail_column(p) + kWidth - 1) / kWidth; }

}  // namespace

// The two forms give the same bits and are compared by what they cost, in us beyond the general kernel's start. A panel's CTA passes over 128 x 128 sub-tiles of its
// row tiles, as many as a CTA of the widest panel has, whatever is left of the last panel and of the SMs that the number of panels does not divide; the general kernel takes waves of
// tiles over all SMs. General / panel, measured: 262144 x 1537 x 512 204 / 174 (rank 1), 16384 x 1345 x 448 15.3 / 15.0, 8192 x 1537 x 512 9.9 / 10.1; last panel
// nearly empty: 65536 x 577 x 192 22.8 / 24.2, 75776 x 288 x 128 12.3 / 16.5; idle SMs: 1024 x 19200 x 512 12.4 / 18.5, 2048 x 12800 x 512 14.9 / 18.6; one half: 151552 x 96 x
// 512 11.1 / 14.5. Over 290 shapes of 384 to 568320 rows, 64 to 24576 columns and K 64 to 512 the choice costs 0.4 % on average against the better of the two, and 9 % at most where it
// takes the panel (by three row tiles per CTA alone 2.5 % and 55 %).
bool gemm_panel_applies(const GemmParams& p, int rk, int sms) {
    if (p.epilogue != EPI_F16 || p.k > kMaxK || p.b2 != nullptr || p.beta != 0.0f || rk > 1) return false;
    const int panels = panels_of(p);
    if (panels > sms) return false;
    const int m_tiles = (p.m + BM - 1) / BM, per = sms / panels, tiles = (m_tiles + per - 1) / per;
    const bool long_k = p.k > BK, halves = p.n - tail_column(p) > 128;
    const long long waves = (static_cast<long long>(m_tiles) * ((p.n + 127) / 128) + sms - 1) / sms;
    // (2 us where the launch is too long to start early; a panel's set-up; with one panel no two tiles of the general kernel share rows of A in time)
    const float panel_us = 1.2f + (tiles > kEarlyTiles ? 2.0f : 0.0f) + static_cast<float>(tiles) * (halves ? (long_k ? 1.6f : 1.48f) : (long_k ? 1.05f : 0.85f));
    const float general_us = (waves > 12 ? 2.0f : 0.0f) + static_cast<float>(waves) * (long_k ? 1.12f : panels == 1 ? 1.2f : 0.9f);
    return panel_us < general_us;
}

int gemm_panel_launch(const GemmParams& p, int rk, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& md, uint32_t group_magic, int sms, int dev,
                      cudaStream_t stream) {
    PanelArgs args;
    args.p = p;
    args.k_atoms = sf_k_atoms(p.k);
    args.group_magic = group_magic;
    args.m_tiles = (p.m + BM - 1) / BM;
    args.tail = tail_column(p);
    args.panels = panels_of(p);
    args.per = std::min(sms / args.panels, args.m_tiles);
    CUtensorMap mbt = mb;
    if (args.tail) {
        const int rc = make_map_2d(&mbt, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.b, static_cast<uint64_t>(p.k) / 2, static_cast<uint64_t>(p.n), static_cast<uint64_t>(p.k) / 2, 128, kTailRows, "B (tail)");
        if (rc) return rc;
    }
    return rk == 0 ? launch_t<0>(ma, mb, mbt, md, args, dev, stream) : launch_t<1>(ma, mb, mbt, md, args, dev, stream);
}

int gemm_panel_device_error(int* code) { return take_wait_error(code); }

}  // namespace bnf4
