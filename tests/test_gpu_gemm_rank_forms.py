"""The rank term of the block-scaled GEMM: every rank, with members whose pairs end inside a warp's 32 rows, between them and never.

The reference is the GEMM without a rank term that adds the term as its C operand. With a scale that is a power of two the term is exact in fp32 (an
integer below 2^24 times the scale), so both round the same sum once: every output is the same bit for bit."""
import pytest

pytestmark = pytest.mark.gpu

EPILOGUES = ["f32", "f16", "add_i8", "gelu_i8", "gelu_fp4"]


def _run(epilogue, resid, next_tvec, **kw):
    import torch
    from bitnet_nvfp4_b200 import host
    m, n = kw["m"], kw["n"]
    if epilogue == "f32":
        d = torch.full((m, n), -7.0, device="cuda")
        host.gemm_nvfp4_ex(epilogue=host.EPI_F32, d=d, ldd=n, **kw)
        return (d,)
    if epilogue == "f16":
        d = torch.full((m, n), -7.0, dtype=torch.float16, device="cuda")
        host.gemm_nvfp4_ex(epilogue=host.EPI_F16, d_f16=d, ld_f16=n, n_f16=n, **kw)
        return (d,)
    if epilogue == "add_i8":
        x = resid.clone()
        host.gemm_nvfp4_ex(epilogue=host.EPI_ADD_I8, resid=x, ld_resid=n, add_scale=1.0, **kw)
        return (x,)
    d8 = torch.full((m, n), -7, dtype=torch.int8, device="cuda")
    if epilogue == "gelu_i8":
        host.gemm_nvfp4_ex(epilogue=host.EPI_GELU_I8, act_scale=0.9, d_i8=d8, ld_i8=n, **kw)
        return (d8,)
    codes, sf = (torch.zeros(b, dtype=torch.uint8, device="cuda") for b in (host.matrix_bytes(m, n), host.sf_bytes(m, n)))
    nvec = next_tvec.shape[1]
    t = torch.zeros(m + 1, max(nvec, 1), dtype=torch.int32, device="cuda")
    if nvec:
        kw.update(next_tvec=next_tvec, next_tvec_pair_stride=nvec * n, next_nvec=nvec, next_t=t)
    host.gemm_nvfp4_ex(epilogue=host.EPI_GELU_FP4, act_scale=0.9, d_codes=codes, d_sf=sf, d_i8=d8, ld_i8=n, **kw)
    return d8, codes, sf, t


@pytest.mark.parametrize("m,n,k,rpm", [
    (400, 160, 192, 48),     # pairs of 96 rows: every warp inside one
    (300, 96, 128, 100),     # pairs end inside a warp
    (330, 288, 128, 5),      # four pairs in a warp
    (257, 64, 64, 0),        # one set of factors for all rows
    (384, 128, 256, 128),    # the batched driver's layout
    (18700, 512, 4096, 1100),  # many K blocks and waves
    (16640, 512, 4096, 2080),
])
@pytest.mark.parametrize("rank,nvec", [(1, 1), (1, 0), (2, 2), (2, 4), (3, 3), (4, 4), (4, 1)])
def test_rank_term_is_an_exact_c_operand(m, n, k, rpm, rank, nvec):
    import torch
    from bitnet_nvfp4_b200 import host
    g = torch.Generator(device="cuda").manual_seed(m + rank)
    pairs = (m + 2 * rpm - 1) // (2 * rpm) if rpm else 1

    def ints(low, high, *shape):
        return torch.randint(low, high, shape, device="cuda", generator=g)

    a, sfa = host.nvfp4_quantize_a(ints(-127, 128, m, k).to(torch.int8))
    b, sfb = host.nvfp4_quantize_b(ints(-1, 2, n, k).to(torch.int8))
    t, A = ints(-1000, 1001, m, rank).int(), ints(-4, 5, pairs, n, rank).to(torch.int8)
    resid, next_tvec = ints(-127, 128, m, n).to(torch.int8), ints(-4, 5, pairs, nvec, n).to(torch.int8)
    scale = 2.0 ** -7
    member = torch.arange(m, device="cuda") // rpm if rpm else torch.zeros(m, dtype=torch.long, device="cuda")
    sign = 1 - 2 * (member % 2)
    term = torch.empty(m, n, device="cuda")
    for p in range(pairs):
        rows = member // 2 == p
        term[rows] = (t[rows].double() @ A[p].double().T * sign[rows, None] * scale).float()
    common = dict(a=a, b=b, sfa=sfa, sfb=sfb, m=m, n=n, k=k, alpha=2.0 ** -5 / k ** 0.5)
    for epilogue in EPILOGUES:
        nt = next_tvec if epilogue == "gelu_fp4" else None
        got = _run(epilogue, resid, nt, rank=rank, rows_per_member=rpm, lora_t=t, t_stride=rank, lora_A=A, lora_A_pair_stride=n * rank, lora_scale=scale, **common)
        want = _run(epilogue, resid, next_tvec[:, :0], c=term, ldc=n, beta=1.0, **common)
        if epilogue == "gelu_fp4":
            sums = torch.zeros_like(got[3])
            if nvec:
                for p in range(pairs):
                    rows = torch.nonzero(member // 2 == p).squeeze(1)
                    sums[rows] = (want[0][rows].double() @ next_tvec[p].double().T).int()
            want = (*want[:3], sums)
        for x, y in zip(got, want):
            assert torch.equal(x, y), epilogue
