"""Row quantisers whose fp32 (or fp16) rows lie on 32-byte, on 16-byte and on 4-byte boundaries, and rows of one, two and four blocks a lane:
the bytes of the normalisation are those of the general kernel over the residual rows."""
import pytest

pytestmark = pytest.mark.gpu


def _shifted(t, elems):
    """A copy of t that starts `elems` elements behind an allocation's first."""
    import torch
    buf = torch.empty(t.numel() + elems, dtype=t.dtype, device=t.device)
    buf[elems:] = t.reshape(-1)
    return buf[elems:].view(t.shape)


@pytest.mark.parametrize("cols,rpm,nvec", [
    (512, 64, 1), (512, 64, 4),   # one block a lane, with the sizes and projections of the batched driver
    (48, 19, 0),                  # most lanes idle
    (528, 19, 5),                 # a second block for one lane, rows per member and columns not powers of two
    (1024, 64, 4), (1040, 19, 2),
    (2048, 19, 16), (2048, 64, 3),
])
@pytest.mark.parametrize("fe", ["act", "pos", "add", "add_half"])
def test_rows_on_every_boundary(fe, cols, rpm, nvec):
    import torch
    from bitnet_nvfp4_b200 import host
    members, T = 4, 16
    rows, pairs = members * rpm, members // 2
    g = torch.Generator(device="cuda").manual_seed(cols + rpm)
    x0 = torch.randint(-127, 128, (rows, cols), device="cuda", generator=g).to(torch.int8)
    f = torch.randn(rows, cols, device="cuda", generator=g) * 30
    pos = torch.randn(T, cols, device="cuda", generator=g)
    noise = torch.randint(-127, 128, (pairs, T, cols), device="cuda", generator=g).to(torch.int8)
    tvec = torch.randint(-127, 128, (pairs, max(nvec, 1), cols), device="cuda", generator=g).to(torch.int8)
    if fe == "add_half":
        f = f.half()

    def outputs():
        return (torch.zeros(host.matrix_bytes(rows, cols), dtype=torch.uint8, device="cuda"), torch.zeros(host.sf_bytes(rows, cols), dtype=torch.uint8, device="cuda"),
                torch.zeros(rows, max(nvec, 1), dtype=torch.int32, device="cuda"))

    def run(front_end, **kw):
        codes, sf, t = outputs()
        if nvec:
            kw.update(tvec=tvec, tvec_pair_stride=nvec * cols, nvec=nvec, t_out=t)
        host.rowquant(front_end, rows=rows, cols_in=cols, cols_out=cols, rows_per_member=rpm, out_codes=codes, out_sf=sf, ld_in=cols, **kw)
        return codes, sf, t

    shifts = {4: (0, 4, 1), 2: (0, 8)}[f.element_size()] if not fe == "add" else (0, 4)  # (the residual add refuses rows off a 16-byte boundary)
    got = []
    for s in shifts:
        fs, x = _shifted(f, s), x0.clone()
        if fe == "act":
            got.append((*run(host.FE_ACT, in_f32=fs, act_mode=3, act_scale=0.9), x))
        elif fe == "pos":
            got.append((*run(host.FE_POS_GELU_ABSMEAN, in_f32=fs, pos=_shifted(pos, s), pos_mod=T, pos_noise=noise, noise_pair_stride=T * cols, sigma=0.125,
                             act_scale=0.9, norm_scale=40.0, inout_i8=x), x))
        else:
            got.append((*run(host.FE_ADD_ABSMEAN, in_f32=fs, in_f16=int(fe == "add_half"), add_scale=1.0, norm_scale=40.0, inout_i8=x), x))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
    codes, sf, t, x = got[0]
    if fe in ("add", "add_half"):
        assert torch.equal(x, (x0.float() + f.float().round()).clamp(-127, 127).to(torch.int8))
    if fe != "act":  # rows off a 16-byte boundary take the general kernel
        ref = run(host.FE_ABSMEAN, in_i8=_shifted(x, 1), norm_scale=40.0)
        fast = run(host.FE_ABSMEAN, in_i8=x, norm_scale=40.0)
        assert all(torch.equal(a, b) for a, b in zip(ref, fast))
        assert all(torch.equal(a, b) for a, b in zip(ref, (codes, sf, t)))


@pytest.mark.parametrize("cols,rpm", [(512, 5376), (1024, 2688)])
@pytest.mark.parametrize("nvec", [1, 16])
@pytest.mark.parametrize("fe", ["act", "add"])
def test_rows_that_fill_much_of_l2(fe, cols, rpm, nvec):
    """fp32 rows of 40 MB and more give the bytes of their halves."""
    import torch
    from bitnet_nvfp4_b200 import host
    g = torch.Generator(device="cuda").manual_seed(cols + nvec)
    x0 = torch.randint(-127, 128, (4 * rpm, cols), device="cuda", generator=g).to(torch.int8)
    f = torch.randn(4 * rpm, cols, device="cuda", generator=g) * 30
    tvec = torch.randint(-127, 128, (2, nvec, cols), device="cuda", generator=g).to(torch.int8)

    def run(pairs):
        rows, part = 2 * rpm * len(pairs), slice(2 * rpm * pairs[0], 2 * rpm * (pairs[-1] + 1))
        codes, sf = (torch.zeros(b, dtype=torch.uint8, device="cuda") for b in (host.matrix_bytes(rows, cols), host.sf_bytes(rows, cols)))
        t, x, y = torch.zeros(rows, nvec, dtype=torch.int32, device="cuda"), x0[part].clone(), f[part].clone()
        kw = dict(in_f32=y, act_mode=3, act_scale=0.9) if fe == "act" else dict(in_f32=y, add_scale=1.0, norm_scale=40.0, inout_i8=x)
        host.rowquant(host.FE_ACT if fe == "act" else host.FE_ADD_ABSMEAN, rows=rows, cols_in=cols, cols_out=cols, rows_per_member=rpm, out_codes=codes, out_sf=sf,
                      ld_in=cols, tvec=tvec[pairs[0]:].contiguous(), tvec_pair_stride=nvec * cols, nvec=nvec, t_out=t, **kw)
        return codes, sf, t, x

    for whole, a, b in zip(run([0, 1]), run([0]), run([1])):
        assert torch.equal(whole, torch.cat([a, b]))
