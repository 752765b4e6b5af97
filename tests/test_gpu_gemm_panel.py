"""The panel form of the block-scaled GEMM (half outputs, K of at most 512, eight row tiles per CTA) against the general kernel.

A call over all rows runs the panel form; the same rows in slices too short for it run the general one, which the other GEMM tests hold to the
oracle. Both accumulate the same products in the same order and round alike: outputs are compared bit for bit. Sizes put the edges
everywhere: a single column behind whole panels, panels of one half or a part of one, K remainders, rows that end inside a tile, pairs that change with
every tile or between them, groups that end inside a panel."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import torch
    from bitnet_nvfp4_b200 import host
    assert torch.cuda.is_available()
    return host


@pytest.mark.parametrize("m,n,k,rank,rpm,group", [
    (32768, 1537, 512, 1, 4096, 512),   # the model's projection: a column behind six panels
    (32741, 1537, 320, 0, 4096, 0),     # rows end inside a tile, K remainder of 64
    (40832, 961, 320, 1, 128, 320),     # members of one tile, groups end inside panels, the fp32 column in the last panel
    (40001, 673, 192, 0, 200, 0),       # the last panel is half a panel and a part, with one fp32 column
    (160000, 129, 64, 1, 128, 0),       # one panel: the fp32 column in its second half, one K block
    (159872, 96, 512, 1, 128, 0),       # three chunks of one half
    (40832, 931, 512, 0, 128, 0),       # three fp32 columns
    (75776, 512, 448, 1, 256, 256),     # two whole panels, a group each
    (75776, 480, 192, 1, 256, 160),     # three groups, and chunks of the last panel behind the third: t has no fourth column for them
    (160000, 96, 64, 1, 128, 32),       # the same with a panel of one half
    (160000, 160, 128, 1, 128, 32),     # a group per chunk, the last half has one of four
])
def test_panel_form_equals_the_general_kernel(H, m, n, k, rank, rpm, group):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, sfa = H.nvfp4_quantize_a(torch.randint(-127, 128, (m, k), device="cuda", generator=g, dtype=torch.int8))
    b, sfb = H.nvfp4_quantize_b(torch.randint(-1, 2, (n, k), device="cuda", generator=g, dtype=torch.int8))
    r, groups = max(rank, 1), -(-n // group) if group else 1
    pairs = -(-m // (2 * rpm))
    A = torch.randint(-4, 5, (pairs, n, r), device="cuda", generator=g, dtype=torch.int8)
    t = torch.randint(-1000, 1000, (m, r * groups), device="cuda", generator=g, dtype=torch.int32)
    n16 = n // 32 * 32
    step = math.lcm(2 * rpm, 128)
    step *= max(1, 2560 // step)
    results = []
    for rows_at_once in (m, step):
        d16 = torch.full((m, n16), 7.0, dtype=torch.float16, device="cuda")
        tail = torch.full((m, max(1, n - n16)), 7.0, device="cuda")
        for r0 in range(0, m, rows_at_once):
            kw = dict(a=a[r0 * k // 2:], b=b, sfa=sfa[H.sf_bytes(r0, k):], sfb=sfb, m=min(rows_at_once, m - r0), n=n, k=k, alpha=0.03, epilogue=H.EPI_F16,
                      d_f16=d16[r0:], ld_f16=n16, n_f16=n16, d=tail[r0:], ldd=max(1, n - n16))
            if rank:
                kw.update(rank=rank, rows_per_member=rpm, lora_t=t[r0:], t_stride=rank * groups, lora_A=A[r0 // (2 * rpm):], lora_A_pair_stride=n * rank,
                          lora_scale=0.01, group_cols=group)
            H.gemm_nvfp4_ex(**kw)
        results.append((d16, tail))
    assert H.device_error() == 0
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
