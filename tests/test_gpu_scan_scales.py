"""Closed-form scan of wide heads where its power-of-two scales of the rows of q and k, taken from the first 32 columns, do not hold for the whole row (they are then taken again),
and at the edges of its blocks: 32 columns of q and k, 64 of v, 16 tokens. Against the recurrence in float64: an inner
product of two rows of unit length is off by up to 3 * 2^-22 (two operands of 22 bits, the product of their low halves left out), and with a cosine of a tenth, as single tokens
have it, that is 2^-17 of the output (seen: 3e-6 at 128 tokens, 1e-6 at one)."""
import pytest

pytestmark = pytest.mark.gpu


def recurrence(q, k, v, logit, method, eps):
    import torch
    q, k, v = q.double(), k.double(), v.double()
    beta, S, out = torch.sigmoid(logit.double()), torch.zeros(q.shape[0], q.shape[2], q.shape[2], dtype=torch.float64, device=q.device), []
    for t in range(q.shape[1]):
        kt, b = k[:, t], beta[:, t]
        lam = (kt * kt).sum(-1).clamp(min=eps)
        if method == 0:
            kt, alpha = kt * (lam + eps).rsqrt()[:, None], b
        else:
            alpha = -torch.expm1(-(b * lam)) / (lam + eps)
        S = S + torch.einsum("ni,nj->nij", kt, alpha[:, None] * (v[:, t] - torch.einsum("nij,ni->nj", S, kt)))
        out.append(torch.einsum("nij,ni->nj", S, q[:, t] * ((q[:, t] ** 2).sum(-1, keepdim=True) + eps).rsqrt()))
    return torch.stack(out, 1)


@pytest.mark.parametrize("method", [1, 0])
@pytest.mark.parametrize("T,hd,kind", [(128, 512, "plain"), (1, 64 + 32, "plain"), (17, 160, "plain"), (113, 288, "plain"), (40, 512, "grow"), (128, 96, "grow"), (40, 320, "shrink"),
                                       (33, 512, "zero first"), (50, 224, "zero rows"), (64, 512, "large"), (64, 512, "small"), (128, 128, "one row"),
                                       (64, 512, "tiny q"), (64, 512, "tiny k"), (40, 96, "tiny q"), (40, 96, "tiny k"), (33, 512, "tinier first"), (33, 512, "tiny")])
def test_scales(T, hd, kind, method):
    import torch
    from bitnet_nvfp4_b200 import host
    seqs = 3
    g = torch.Generator(device="cuda").manual_seed(T + hd + method)
    q, k, v = (torch.randn(seqs, T, hd, device="cuda", generator=g) * 0.3 for _ in range(3))
    ramp = torch.exp2(torch.linspace(-12, 12, hd, device="cuda"))
    if kind == "grow":
        q, k = q * ramp, k * ramp * 1e-3
    elif kind == "shrink":
        q, k = q * ramp.flip(0), k * ramp.flip(0) * 1e-3
    elif kind == "zero first":
        q[..., :32] = 0
        k[..., :64] = 0
    elif kind == "zero rows":
        k[:, ::3] = 0
        q[:, 1::4] = 0
    elif kind == "large":
        q, k = q * 1e15, k * 1e15
    elif kind == "small":
        q, k = q * 1e-5, k * 1e-17
    elif kind == "tiny q":  # squares that underflow, behind a scale of 2^107
        q[:, 1::4] *= 1e-24
        q[:, 1::4, :32] *= 1e-6
    elif kind == "tiny k":
        k[:, ::3] *= 1e-24
        k[:, ::3, :32] *= 1e-6
    elif kind == "tinier first":
        q[:, 1::4, :32] *= 1e-30
        k[:, ::3, :32] *= 1e-30
    elif kind == "tiny":
        q[:, 1::4] *= 1e-36
        k[:, ::3] *= 1e-36
    elif kind == "one row":
        q[1, 100, 70] = 3e4  # (out of the range of the first columns' scale)
        k[2, 64, 127] = -7e5
    logit = torch.randn(seqs, T, device="cuda", generator=g)
    qkv = torch.cat([q, k, v], -1).reshape(seqs * T, 3 * hd).contiguous()
    out = torch.empty(seqs * T, hd, device="cuda")
    host.efla_scan(state=None, state_fp16=1, q=qkv, k=qkv[:, hd:], v=qkv[:, 2 * hd:], beta_raw=logit.reshape(-1), ld_qkv=3 * hd, ld_beta=1, beta_bias=0.0, seqs_per_bias=1,
                   hidden=hd, heads=1, seqs=seqs, T=T, method=method, eps=1e-6, out=out, ld_out=hd, variant=0, qkv_f16=0, out_f16=0)
    assert host.device_error() == 0
    want = recurrence(q, k, v, logit, method, 1e-6)
    err = (out.reshape(seqs, T, hd).double() - want).abs().amax((1, 2))
    assert (err <= 2.0 ** -17 * want.abs().amax((1, 2))).all(), (err / want.abs().amax((1, 2))).tolist()


@pytest.mark.parametrize("norm", [0.01, 0.26, 0.9, 20.0])
@pytest.mark.parametrize("T,hd", [(33, 512), (128, 256), (64, 96), (50, 224)])
def test_zeros_first_cost_no_bits(T, hd, norm):
    """Rows whose first 32 columns are zero are off by what the same rows with these columns last are off by: the products are the same, their
    sums begin at another column. (Seen: within 5e-5 of each other; 1.5 to 1.8 times as much where rows of norm 0.26 were left unscaled.)"""
    import torch
    from bitnet_nvfp4_b200 import host
    seqs = 24
    g = torch.Generator(device="cuda").manual_seed(T + hd)
    q, k, v = (torch.randn(seqs, T, hd, device="cuda", generator=g) for _ in range(3))
    for x in (q, k):
        x[..., hd - 32:] = 0
        x *= norm / x.norm(dim=-1, keepdim=True)
    logit = torch.randn(seqs, T, device="cuda", generator=g)
    want = recurrence(q, k, v, logit, 1, 1e-6)
    err = []
    for shift in (0, 32):
        qkv = torch.cat([q.roll(shift, -1), k.roll(shift, -1), v], -1).reshape(seqs * T, 3 * hd).contiguous()
        out = torch.empty(seqs * T, hd, device="cuda")
        host.efla_scan(state=None, state_fp16=1, q=qkv, k=qkv[:, hd:], v=qkv[:, 2 * hd:], beta_raw=logit.reshape(-1), ld_qkv=3 * hd, ld_beta=1, beta_bias=0.0, seqs_per_bias=1,
                       hidden=hd, heads=1, seqs=seqs, T=T, method=1, eps=1e-6, out=out, ld_out=hd, variant=0, qkv_f16=0, out_f16=0)
        err.append(float((out.reshape(seqs, T, hd).double() - want).norm()))
    assert err[1] <= 1.01 * err[0], err


def test_values_that_are_no_numbers_behind_the_first_columns():
    """An infinite q meets its own row, an infinite k cuts the sequence, a norm that overflows leaves the state alone; rows of other sequences keep their bits."""
    import torch
    from bitnet_nvfp4_b200 import host
    seqs, T, hd = 4, 48, 192
    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(seqs, T, hd, device="cuda", generator=g) * 0.3 for _ in range(3))
    logit = torch.randn(seqs, T, device="cuda", generator=g)

    def run():
        qkv = torch.cat([q, k, v], -1).reshape(seqs * T, 3 * hd).contiguous()
        out = torch.empty(seqs * T, hd, device="cuda")
        host.efla_scan(state=None, state_fp16=1, q=qkv, k=qkv[:, hd:], v=qkv[:, 2 * hd:], beta_raw=logit.reshape(-1), ld_qkv=3 * hd, ld_beta=1, beta_bias=0.0, seqs_per_bias=1,
                       hidden=hd, heads=1, seqs=seqs, T=T, method=1, eps=1e-6, out=out, ld_out=hd, variant=0, qkv_f16=0, out_f16=0)
        assert host.device_error() == 0
        return out.reshape(seqs, T, hd)
    base = run()
    q[0, 20, 150] = float("inf")
    k[1, 30, 100] = float("inf")
    k[2, 10, 64:] = 1e25  # finite, |k|^2 is not
    got = run()
    assert torch.equal(got[3], base[3])
    assert torch.isnan(got[0, 20]).all() and not torch.isnan(got[0, :20]).any() and not torch.isnan(got[0, 21:]).any()
    other = torch.arange(T, device="cuda") != 20
    assert (got[0][other] - base[0][other]).abs().max() <= 2.0 ** -17 * base[0].abs().max()  # (the unit's rows take their scales from whole rows then)
    assert torch.isnan(got[1, 30:]).all() and (got[1, :30] - base[1, :30]).abs().max() <= 2.0 ** -17 * base[1].abs().max()
    assert not torch.isnan(got[2]).any() and (got[2, :10] - base[2, :10]).abs().max() <= 2.0 ** -17 * base[2].abs().max()
