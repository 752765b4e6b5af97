"""Row quantisers with more than four projections: several rows per warp, whose projections are taken together."""
import numpy as np
import pytest

import oracle_lib as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,hid,nvec,rpm", [
    (37891, 320, 16, 17),     # pairs end inside a batch of eight rows; the last batch has three; a tail of the columns
    (37889, 512, 7, 1),       # two rows per pair; a last batch of one row; one half of the vectors' operand empty
    (28420, 1024, 9, 14210),  # two blocks per lane, one vector in the second half
    (9602, 2048, 5, 4801),    # four rows per batch, a group of one vector
    (9603, 1536, 13, 5),      # idle lanes in the last block; pairs end inside a batch; a last batch of three rows
    (37888, 16, 12, 0),       # one block per row, one set of vectors for all rows
    (50, 512, 12, 3),         # too few rows for batches
])
def test_more_than_four_projections(rows, hid, nvec, rpm):
    import torch
    from bitnet_nvfp4_b200 import host as H
    rng = np.random.default_rng(rows + hid)
    pairs = (rows + 2 * rpm - 1) // (2 * rpm) if rpm else 1
    x = rng.integers(-127, 128, (rows, hid)).astype(np.int8)
    tvec = rng.integers(-127, 128, (pairs, nvec, hid)).astype(np.int8)
    xd, tv = torch.from_numpy(x).cuda(), torch.from_numpy(tvec).cuda()
    yq = torch.zeros((rows, hid), dtype=torch.int8, device="cuda")
    codes = torch.zeros(rows * hid // 2, dtype=torch.uint8, device="cuda")
    sf = torch.zeros(H.sf_bytes(rows, hid), dtype=torch.uint8, device="cuda")
    t = torch.full((rows + 1, nvec), -7, dtype=torch.int32, device="cuda")
    H.rowquant(H.FE_ABSMEAN, rows=rows, cols_in=hid, cols_out=hid, rows_per_member=rpm, in_i8=xd, ld_in=hid, norm_scale=40.0, out_q=yq,
               ld_q=hid, out_codes=codes, out_sf=sf, tvec=tv, tvec_pair_stride=nvec * hid, nvec=nvec, t_out=t)
    q, c, s = orc.absmean_norm_q(x.copy(), None, 0.0, 40.0)
    assert np.array_equal(yq.cpu().numpy(), q)
    assert np.array_equal(codes.cpu().numpy(), np.asarray(c).reshape(-1)) and np.array_equal(sf.cpu().numpy(), np.asarray(s).reshape(-1))
    pair = np.arange(rows) // (2 * rpm) if rpm else np.zeros(rows, int)
    ref = np.empty((rows, nvec), np.int32)
    for p in range(pairs):
        ref[pair == p] = q[pair == p].astype(np.int32) @ tvec[p].astype(np.int32).T
    got = t.cpu().numpy()
    assert np.array_equal(got[:rows], ref)
    assert (got[rows] == -7).all()


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("scale", [1.0, 0.8, 1000.0])
def test_non_finite_activations_do_not_depend_on_alignment(mode, scale):
    """Rows on a 16-byte boundary take the vectorised kernel, others the general one; NaN becomes 0 in both."""
    import torch
    from bitnet_nvfp4_b200 import host
    rows, cols = 40, 512
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(rows, cols, device="cuda", generator=g) * 3
    special = torch.tensor([float("nan"), float("inf"), float("-inf"), 3e38, -3e38, 1e-40, -0.0, float("nan")], device="cuda")
    at = torch.randperm(rows * cols, device="cuda", generator=g)[:400]
    x.view(-1)[at] = special[torch.arange(400, device="cuda") % 8]
    buf = torch.empty(rows * cols + 1, device="cuda")
    buf[1:] = x.view(-1)
    outs = []
    for t in (x, buf[1:].view(rows, cols)):
        q = torch.empty(rows, cols, dtype=torch.int8, device="cuda")
        codes, sf = torch.zeros(host.matrix_bytes(rows, cols), dtype=torch.uint8, device="cuda"), torch.zeros(host.sf_bytes(rows, cols), dtype=torch.uint8, device="cuda")
        host.rowquant(host.FE_ACT, rows=rows, cols_in=cols, cols_out=cols, in_f32=t, ld_in=cols, act_mode=mode, act_scale=scale, out_q=q, ld_q=cols, out_codes=codes, out_sf=sf)
        outs.append((q, codes, sf))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
    assert not outs[0][0].view(-1)[at][torch.arange(400, device="cuda") % 8 == 0].any()
