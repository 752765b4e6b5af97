"""CTA-pair instances of the block-scaled GEMM (long K, enough waves of 256 x 256 tiles to pay) against the single-CTA instances.

A call over all rows runs the pair instance; the same rows in slices too small for it run the single-CTA one, which the other GEMM
tests hold to the oracle. Both accumulate the same MMAs in the same order and share the epilogue code: outputs are compared bit for
bit. Sizes put the edges everywhere: rows that end inside the first or the second CTA's half of the last tile, columns that end
inside either 128-column half, a K remainder of 64."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import torch
    from bitnet_nvfp4_b200 import host
    assert torch.cuda.is_available()
    return host


# rows of a slice: whole pairs of members, multiples of 128 (scale atoms), too few for the pair instance
@pytest.mark.parametrize("m,n,k,rank,rpm,slice_rows", [
    (69120, 768, 1024, 1, 128, 1280),     # the model's instance: rank 1, tiles inside one member, m a multiple of 256
    (69220, 640, 1088, 0, 0, 1280),       # ends in the first CTA's half; the last tile column is half a tile
    (68300, 736, 1600, 2, 640, 1280),     # ends in the second CTA's half; 736 = 2 x 256 + 224; members straddle tiles
    (96200, 513, 2112, 4, 320, 1280),     # one column in the third tile column (fp32 / half only)
    (37632, 768, 2048, 1, 128, 1280),     # GELU's threshold
    (96000, 512, 2112, 4, 640, 1280),
])
def test_pair_instance_equals_single_cta_instance(H, m, n, k, rank, rpm, slice_rows):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, sfa = H.nvfp4_quantize_a(torch.randint(-127, 128, (m, k), device="cuda", generator=g, dtype=torch.int8))
    b, sfb = H.nvfp4_quantize_b(torch.randint(-1, 2, (n, k), device="cuda", generator=g, dtype=torch.int8))
    r = max(rank, 1)
    pairs = (m + 2 * rpm - 1) // (2 * rpm) if rank else 1
    A = torch.randint(-4, 5, (pairs, n, r), device="cuda", generator=g, dtype=torch.int8)
    t = torch.randint(-1000, 1000, (m, r), device="cuda", generator=g, dtype=torch.int32)
    tv = torch.randint(-4, 5, (pairs, r, n), device="cuda", generator=g, dtype=torch.int8)
    resid0 = torch.randint(-100, 101, (m, n), device="cuda", generator=g, dtype=torch.int8)
    c = torch.randn(m, n, device="cuda", generator=g)
    n16 = n // 32 * 32
    epilogues = [H.EPI_F32] + ([H.EPI_F16] if n16 else [])
    if n % 32 == 0:
        epilogues += [H.EPI_ADD_I8] + ([H.EPI_GELU_I8, H.EPI_GELU_FP4] if k >= 2048 else [])
    for epi in epilogues:
        results = []
        for step in (m, slice_rows):
            d = torch.zeros(m, n, device="cuda")
            d16, tail = torch.zeros(m, n16, dtype=torch.float16, device="cuda"), torch.zeros(m, max(1, n - n16), device="cuda")
            resid, d8 = resid0.clone(), torch.zeros(m, n, dtype=torch.int8, device="cuda")
            codes, sf = torch.zeros(m, n // 2, dtype=torch.uint8, device="cuda"), torch.zeros(H.sf_bytes(m, n), dtype=torch.uint8, device="cuda")
            nt = torch.zeros(m, r, dtype=torch.int32, device="cuda")
            for r0 in range(0, m, step):
                rows = min(step, m - r0)
                kw = dict(a=a[r0 * k // 2:], b=b, sfa=sfa[H.sf_bytes(r0, k):], sfb=sfb, m=rows, n=n, k=k, alpha=0.03, epilogue=epi)
                p0 = r0 // (2 * rpm) if rank else 0
                if rank:
                    kw.update(rank=rank, rows_per_member=rpm, lora_t=t[r0:], t_stride=rank, lora_A=A[p0:], lora_A_pair_stride=n * rank, lora_scale=0.01)
                elif epi == H.EPI_F32:
                    kw.update(beta=0.5, c=c[r0:], ldc=n)
                if epi == H.EPI_F32:
                    kw.update(d=d[r0:], ldd=n)
                elif epi == H.EPI_F16:
                    kw.update(d_f16=d16[r0:], ld_f16=n16, n_f16=n16, d=tail[r0:], ldd=max(1, n - n16))
                elif epi == H.EPI_ADD_I8:
                    kw.update(resid=resid[r0:], ld_resid=n, add_scale=0.07)
                elif epi == H.EPI_GELU_I8:
                    kw.update(act_scale=4.0, d_i8=d8[r0:], ld_i8=n)
                else:
                    kw.update(act_scale=4.0, d_codes=codes[r0:], d_sf=sf[H.sf_bytes(r0, n):])
                    if rank:
                        kw.update(next_tvec=tv[p0:], next_tvec_pair_stride=rank * n, next_nvec=rank, next_t=nt[r0:])
                H.gemm_nvfp4_ex(**kw)
            assert H.device_error() == 0
            results.append((d, d16, tail, resid, d8, codes, sf, nt))
        for whole, parts in zip(*results):
            assert torch.equal(whole, parts), epi
