"""The panel form of the block-scaled GEMM (half outputs, K of at most 512, several row tiles per CTA) against the general kernel.

A call over all rows runs the panel form; the same rows in slices too short for it run the general one, which the other GEMM tests hold to the
oracle (the profiler says which kernel ran). Both accumulate the same products in the same order and round alike: outputs are compared bit for bit. Sizes put the edges
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


class Kernels:
    """Names of the GEMM kernels that run inside the block."""
    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        self.p = torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA])
        self.p.__enter__()
        return self

    def __exit__(self, *exc):
        import torch
        torch.cuda.synchronize()
        self.p.__exit__(*exc)
        self.names = {n for e in self.p.events() for n in ("gemm_panel_kernel", "gemm_nvfp4_kernel") if n in e.name}
        return False


@pytest.mark.parametrize("m,n,k,rank,rpm,group", [
    (32768, 1537, 512, 1, 1024, 512),   # the model's projection: a column behind six panels
    (32741, 1537, 320, 0, 1024, 0),     # rows end inside a tile, K remainder of 64
    (40832, 961, 320, 1, 128, 320),     # members of one tile, groups end inside panels, the fp32 column in the last panel
    (40001, 673, 192, 0, 200, 0),       # the last panel is half a panel and a part, with one fp32 column
    (160000, 129, 64, 1, 128, 0),       # one panel: the fp32 column in its second half, one K block
    (600064, 96, 512, 1, 128, 0),       # three chunks of one half
    (40832, 931, 512, 0, 128, 0),       # three fp32 columns
    (75776, 512, 448, 1, 256, 256),     # two whole panels, a group each
    (75776, 480, 192, 1, 256, 160),     # three groups, and chunks of the last panel behind the third: t has no fourth column for them
    (400000, 96, 64, 1, 128, 32),       # the same with a panel of one half
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
        calls = []
        for r0 in range(0, m, rows_at_once):
            kw = dict(a=a[r0 * k // 2:], b=b, sfa=sfa[H.sf_bytes(r0, k):], sfb=sfb, m=min(rows_at_once, m - r0), n=n, k=k, alpha=0.03, epilogue=H.EPI_F16,
                      d_f16=d16[r0:], ld_f16=n16, n_f16=n16, d=tail[r0:], ldd=max(1, n - n16))
            if rank:
                kw.update(rank=rank, rows_per_member=rpm, lora_t=t[r0:], t_stride=rank * groups, lora_A=A[r0 // (2 * rpm):], lora_A_pair_stride=n * rank,
                          lora_scale=0.01, group_cols=group)
            calls.append(kw)
        with Kernels() as ran:
            for kw in calls:
                H.gemm_nvfp4_ex(**kw)
        assert ran.names == {"gemm_panel_kernel" if rows_at_once == m else "gemm_nvfp4_kernel"}
        results.append((d16, tail))
    assert H.device_error() == 0
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("m,n,k,panel", [
    (16384, 1537, 512, True), (32768, 769, 256, True), (18432, 2048, 512, True), (4096, 8224, 512, True),
    (65536, 577, 192, False), (75776, 288, 128, False),                              # little is left for the last panel's CTAs
    (2048, 12800, 512, False), (1024, 19200, 512, False), (384, 24576, 128, False),  # a third to a half of the SMs would idle
    (151552, 96, 512, False),                                                        # passes of one half
    (2048, 1537, 512, False),                                                        # one row tile per CTA
])
def test_the_cheaper_form_runs(H, m, n, k, panel):
    import torch
    a, sfa = H.nvfp4_quantize_a(torch.ones(m, k, device="cuda", dtype=torch.int8))
    b, sfb = H.nvfp4_quantize_b(torch.ones(n, k, device="cuda", dtype=torch.int8))
    n16 = n // 32 * 32
    d16, tail = torch.empty(m, n16, dtype=torch.float16, device="cuda"), torch.empty(m, max(1, n - n16), device="cuda")
    with Kernels() as ran:
        H.gemm_nvfp4_ex(a=a, b=b, sfa=sfa, sfb=sfb, m=m, n=n, k=k, alpha=0.03, epilogue=H.EPI_F16, d_f16=d16, ld_f16=n16, n_f16=n16, d=tail, ldd=max(1, n - n16))
    assert ran.names == {"gemm_panel_kernel" if panel else "gemm_nvfp4_kernel"}
