"""GELU epilogue with FP4 output where its common path ends: blocks that saturate, values on a rounding boundary or that are no numbers, rows
past the matrix in the last tile, one to four projections of the next product for each form of the rank term.

The int8 values are held to the tanh form in float64 of the kernel's own fp32 output (same accumulators). That form in fp32 is within 1e-6 (1 + |v act_scale|)
of it (tanhf 2 ulp, three roundings), so a value that close to a boundary may go either way: blocks with one are left out (and rows, for the projections)."""
import numpy as np
import pytest

import oracle_lib as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,rank,nvec,alpha,act_scale", [
    (256, 128, 64, 1, 1, 0.05, 1.0), (256, 128, 64, 1, 1, 3.7, 1.0), (384, 96, 128, 1, 1, 0.01, 7.5), (256, 64, 64, 1, 1, 0.002, 900.0),
    (200, 96, 64, 4, 4, 0.05, 1.0), (129, 32, 64, 4, 1, 3.7, 1.0), (160, 64, 64, 4, 3, 0.05, 0.3), (100, 64, 64, 4, 0, 0.05, 1.0), (520, 512, 2048, 4, 4, 0.01, 2.9),
    (200, 96, 64, 2, 2, 0.05, 1.0), (130, 64, 64, 0, 0, 3.7, 1.0), (130, 64, 64, 0, 3, 0.05, 31.0)])
def test_gelu_fp4(m, n, k, rank, nvec, alpha, act_scale):
    import torch
    from bitnet_nvfp4_b200 import host as H
    rng = np.random.default_rng(m + n + k + rank + nvec)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    rpm = 128 if rank == 1 else 32
    x = np.clip(np.rint(rng.standard_normal((m, k)) * 40), -127, 127).astype(np.int8)
    a, sfa = H.nvfp4_quantize_a(dev(x))
    b, sfb = H.nvfp4_quantize_b(dev(rng.integers(-1, 2, (n, k)).astype(np.int8)))
    sfa = sfa.clone()
    sfa.view(-1)[5 * 16] = 0x7f  # the scale of row 5's first block is no number
    pairs = (m + 2 * rpm - 1) // (2 * rpm)
    kw = dict(a=a, b=b, sfa=sfa, sfb=sfb, m=m, n=n, k=k, alpha=alpha)
    if rank:
        kw.update(rank=rank, rows_per_member=rpm, lora_t=dev(rng.integers(-300, 300, (m, rank)).astype(np.int32)), t_stride=rank,
                  lora_A=dev(rng.integers(-4, 5, (pairs, n, rank)).astype(np.int8)), lora_A_pair_stride=n * rank, lora_scale=alpha * 0.123)
    elif nvec:
        kw.update(rows_per_member=rpm)
    d = torch.empty((m, n), dtype=torch.float32, device="cuda")
    H.gemm_nvfp4_ex(d=d, ldd=n, epilogue=H.EPI_F32, **kw)
    codes = torch.zeros(H.matrix_bytes(m, n), dtype=torch.uint8, device="cuda")
    sf = torch.zeros(H.sf_bytes(m, n), dtype=torch.uint8, device="cuda")
    tvec = rng.integers(-4, 5, (pairs, max(1, nvec), n)).astype(np.int8)
    guard = 64
    nt = torch.zeros(m * max(1, nvec) + guard, dtype=torch.int32, device="cuda")
    if nvec:
        kw.update(next_tvec=dev(tvec), next_tvec_pair_stride=nvec * n, next_nvec=nvec, next_t=nt)
    H.gemm_nvfp4_ex(epilogue=H.EPI_GELU_FP4, act_scale=act_scale, d_codes=codes, d_sf=sf, **kw)
    assert H.device_error() == 0
    v = d.cpu().numpy().astype(np.float64)
    assert np.isnan(v[5]).all() and not np.isnan(np.delete(v, 5, 0)).any()
    f = 0.5 * v * (1.0 + np.tanh(0.7978845608028654 * (v + 0.044715 * v ** 3))) * float(np.float32(act_scale))
    f[5] = 0.0  # an integer conversion turns NaN into 0
    want = np.clip(np.rint(f), -127, 127).astype(np.int8)
    near = np.abs(np.abs(f - np.rint(f)) - 0.5) < 1e-6 * (1.0 + np.abs(v * act_scale))
    near &= np.abs(f) < 128.0  # (saturated either way)
    near[5] = False
    assert near.mean() < 2e-3
    rc, rs = orc.quantize_rowmajor(want)
    fine = ~near.reshape(m, n // 16, 16).any(2)
    got = codes.cpu().numpy()[: m * n // 2].reshape(m, n // 16, 8)
    assert np.array_equal(got[fine], np.asarray(rc)[: m * n // 2].reshape(m, n // 16, 8)[fine])
    r, kb = np.nonzero(fine)
    at = ((r >> 7) * ((n // 16 + 3) // 4) + (kb >> 2)) * 512 + (r & 31) * 16 + ((r & 127) >> 5) * 4 + (kb & 3)  # 512-byte atoms of 128 rows x 4 blocks
    assert np.array_equal(sf.cpu().numpy()[at], np.asarray(rs)[at])
    t = nt.cpu().numpy()
    assert (t[m * max(1, nvec):] == 0).all()
    if nvec:
        pair = np.arange(m) // (2 * rpm) * (rank > 0)  # (without a rank term there are no members)
        rows = fine.all(1)
        wt = np.einsum("mn,mvn->mv", want.astype(np.int64), tvec[pair].astype(np.int64))
        assert rows.mean() > 0.5 and np.array_equal(t[: m * nvec].reshape(m, nvec)[rows], wt[rows])
