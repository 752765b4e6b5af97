"""Rank-r term of the block-scaled GEMM where pairs of members do not start at multiples of a tile: a warp's 32 rows then belong to two or
more pairs, each with a factor of its own. Against the fp32 product plus the term computed in float64 (the term is an exact integer
times one scale; the sum is rounded once or twice at 2^-24 relative, far below the bound)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [1, 2, 3, 4])
@pytest.mark.parametrize("m,n,rpm", [(777, 96, 37), (300, 161, 1), (1000, 64, 7), (650, 128, 100), (512, 96, 16), (333, 64, 0), (130, 32, 65)])
def test_rank_term_with_members_of_any_length(m, n, rpm, rank):
    import torch
    from bitnet_nvfp4_b200 import host as H
    rng = np.random.default_rng(m + n + rpm + rank)
    k = 64
    a, sfa = H.nvfp4_quantize_a(torch.from_numpy(rng.integers(-127, 128, (m, k)).astype(np.int8)).cuda())
    b, sfb = H.nvfp4_quantize_b(torch.from_numpy(rng.integers(-1, 2, (n, k)).astype(np.int8)).cuda())
    member = np.arange(m) // rpm if rpm else np.zeros(m, int)
    A = rng.integers(-4, 5, (member[-1] // 2 + 1, n, rank)).astype(np.int8)
    t = rng.integers(-3000, 3000, (m, rank)).astype(np.int32)
    base = H.gemm_ternary_f_nvfp4(a, b, sfa, sfb, m, n, k, 0.1).cpu().numpy().astype(np.float64)
    d = torch.empty((m, n), dtype=torch.float32, device="cuda")
    H.gemm_nvfp4_ex(a=a, b=b, sfa=sfa, sfb=sfb, m=m, n=n, k=k, alpha=0.1, d=d, ldd=n, epilogue=H.EPI_F32, rank=rank, rows_per_member=rpm,
                    lora_t=torch.from_numpy(t).cuda(), t_stride=rank, lora_A=torch.from_numpy(A).cuda(), lora_A_pair_stride=n * rank, lora_scale=0.003)
    assert H.device_error() == 0
    sign = np.where(member % 2 == 0, 1.0, -1.0)
    want = base + float(np.float32(0.003)) * sign[:, None] * np.einsum("mr,mnr->mn", t.astype(np.int64), A[member // 2].astype(np.int64))
    assert np.abs(d.cpu().numpy() - want).max() <= 4 * 2.0 ** -24 * np.abs(want).max()
