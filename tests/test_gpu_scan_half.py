"""Closed form of the scan on half inputs and outputs (heads of 64, 33 to 128 tokens, method 1, zero state) against the recurrence in float64, and against
the chunked form.

Its operands are halves (2^-11 relative: a V, U, P, a G, T) with fp32 sums; the chunked form additionally rounds a W and, after every 16 tokens,
the state. The output's own rounding is 2.1e-4 of its norm, the operands' roundings add about as much each in quadrature: 6e-4 in all at
scales where keys interact, and never more than the chunked form, up to the sampling error of the norms (3 %)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [33, 48, 49, 64, 65, 80, 81, 96, 100, 112, 113, 127, 128]


@pytest.fixture(scope="module")
def H():
    import torch
    from bitnet_nvfp4_b200 import host
    assert torch.cuda.is_available()
    return host


def exact(qkv, beta, heads, seqs, T, bias=-2.0, eps=1e-6):
    import torch
    x = qkv[:, :3 * 64 * heads].double().reshape(seqs, T, 3, heads, 64)
    q, k, v = x[:, :, 0], x[:, :, 1], x[:, :, 2]
    b = torch.sigmoid(beta.double().reshape(seqs, T) + bias)
    S = torch.zeros(seqs, heads, 64, 64, dtype=torch.float64, device="cuda")
    out = []
    for t in range(T):
        lam = (k[:, t] * k[:, t]).sum(-1).clamp(min=eps)
        alpha = -torch.expm1(-(b[:, t, None] * lam)) / (lam + eps)
        S = S + torch.einsum("shd,shn->shdn", alpha[..., None] * k[:, t], v[:, t] - torch.einsum("shd,shdn->shn", k[:, t], S))
        out.append(torch.einsum("shd,shdn->shn", q[:, t], S) * torch.rsqrt((q[:, t] * q[:, t]).sum(-1, keepdim=True) + eps))
    return torch.stack(out, 1).reshape(seqs * T, 64 * heads)


def run(H, qkv, beta, heads, seqs, T, variant=0):
    import torch
    hidden = 64 * heads
    out = torch.full((seqs * T, hidden + 8), 7.0, dtype=torch.float16, device="cuda")
    H.efla_scan(state=None, state_fp16=1, q=qkv, k=qkv[:, hidden:], v=qkv[:, 2 * hidden:], beta_raw=beta, ld_qkv=qkv.shape[1], ld_beta=1, beta_bias=-2.0,
                seqs_per_bias=1, hidden=hidden, heads=heads, seqs=seqs, T=T, method=1, eps=1e-6, out=out, ld_out=hidden + 8, variant=variant, qkv_f16=1, out_f16=1)
    assert H.device_error() == 0
    assert bool((out[:, hidden:] == 7.0).all())  # nothing is written beside the output
    return out[:, :hidden]


def inputs(T, heads, seqs, scale):
    import torch
    g = torch.Generator(device="cuda").manual_seed(T * 97 + heads)
    return (torch.randn(seqs * T, 3 * 64 * heads + 16, device="cuda", generator=g) * scale).half(), torch.randn(seqs * T, device="cuda", generator=g) * 2


@pytest.mark.parametrize("T", LENGTHS)
@pytest.mark.parametrize("heads,seqs,scale", [(2, 301, 0.3), (3, 1, 1.0), (1, 40, 0.03)])
def test_closed_form(H, T, heads, seqs, scale):
    qkv, beta = inputs(T, heads, seqs, scale)
    ref = exact(qkv, beta, heads, seqs, T)
    closed, chunked = (float((run(H, qkv, beta, heads, seqs, T, v).double() - ref).norm() / ref.norm()) for v in (0, 3))
    assert closed <= 6e-4
    assert closed <= (1.03 if seqs * heads * T > 2000 else 1.1) * chunked  # (fewer rows: a tenth for the norms' sampling error)


@pytest.mark.parametrize("T", [48, 64, 100, 128])
@pytest.mark.parametrize("q_scale,k_scale,v_scale,decades", [(1.0, 1e-5, 1000.0, 0), (1.0, 1e-4, 100.0, 0), (30.0, 100.0, 100.0, 0), (0.01, 1e3, 1e3, 0), (0.01, 1e4, 1e4, 0),
                                                             (1.0, 10.0, 1.0, 3), (0.01, 10.0, 100.0, 3), (1.0, 0.1, 10.0, 3), (1.0, 100.0, 1e3, 2)])
def test_keys_of_any_length(H, T, q_scale, k_scale, v_scale, decades):
    """Coefficients and the solution are halves whatever the keys' lengths, the same for all tokens or spread over decades: the error is that of keys of
    ordinary length. (Values keep y above fp16's smallest numbers.)"""
    import torch
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(20 * T, 3, 2, 64, device="cuda", generator=g) * torch.tensor([q_scale, k_scale, v_scale], device="cuda")[None, :, None, None]
    x[:, 1] *= 10.0 ** ((torch.rand(20 * T, 1, 1, device="cuda", generator=g) * 2 - 1) * decades)
    qkv = torch.nn.functional.pad(x.clamp(-65504, 65504).half().reshape(20 * T, -1), (0, 16))
    beta = torch.randn(20 * T, device="cuda", generator=g) * 2
    ref = exact(qkv, beta, 2, 20, T)
    assert float((run(H, qkv, beta, 2, 20, T).double() - ref).norm() / ref.norm()) <= 6e-4


@pytest.mark.parametrize("T", [48, 64])
def test_a_sequence_does_not_depend_on_its_tile(H, T):
    """Two sequences share a tile: one with keys of extreme lengths leaves the other's bits alone."""
    import torch
    qkv, beta = inputs(T, 2, 6, 0.3)
    clean = run(H, qkv, beta, 2, 6, T).reshape(6, T, 128)
    for s, factor in ((0, 1e4), (3, 1e-5), (5, 1e4)):
        far = qkv.clone().reshape(6, T, -1)
        far[s, :, 128:256] *= factor
        got = run(H, far.reshape(6 * T, -1), beta, 2, 6, T).reshape(6, T, 128)
        assert not torch.equal(got[s], clean[s])
        assert all(torch.equal(got[i], clean[i]) for i in range(6) if i != s)


@pytest.mark.parametrize("where", [0, 1, 2])
@pytest.mark.parametrize("T", [33, 64, 72, 128])
def test_in_place(H, T, where):
    """An output that lies on q, k or v, for tiles of one and of two sequences."""
    import torch
    qkv, beta = inputs(T, 3, 400, 0.3)
    apart = run(H, qkv, beta, 3, 400, T)
    x = qkv.clone()
    out = x[:, where * 192:]
    H.efla_scan(state=None, state_fp16=1, q=x, k=x[:, 192:], v=x[:, 384:], beta_raw=beta, ld_qkv=x.shape[1], ld_beta=1, beta_bias=-2.0, seqs_per_bias=1, hidden=192,
                heads=3, seqs=400, T=T, method=1, eps=1e-6, out=out, ld_out=x.shape[1], variant=0, qkv_f16=1, out_f16=1)
    assert H.device_error() == 0 and torch.equal(out[:, :192], apart)


@pytest.mark.parametrize("T", [33, 64, 100, 128])
def test_a_sequence_does_not_depend_on_its_company(H, T):
    import torch
    qkv, beta = inputs(T, 2, 200, 0.3)
    whole = run(H, qkv, beta, 2, 200, T)
    for first, count in ((0, 1), (3, 2), (7, 150)):
        part = run(H, qkv[first * T:(first + count) * T], beta[first * T:(first + count) * T], 2, count, T)
        assert torch.equal(part, whole[first * T:(first + count) * T])


@pytest.mark.parametrize("T", [50, 128])
@pytest.mark.parametrize("where", [0, 1, 2])
def test_values_that_are_no_numbers_stay_behind_their_block(H, T, where):
    """Blocks of 16 tokens before such a value come out as without it, and so do other sequences and heads."""
    import torch
    heads, seqs = 2, 5
    qkv, beta = inputs(T, heads, seqs, 0.3)
    clean = run(H, qkv, beta, heads, seqs, T).reshape(seqs, T, heads, 64)
    for s, t, value in ((1, 17, np.nan), (3, T - 1, np.inf), (4, 40, -np.inf)):
        bad = qkv.clone()
        bad[s * T + t, where * 64 * heads + 64 + 5] = value
        got = run(H, bad, beta, heads, seqs, T).reshape(seqs, T, heads, 64)
        assert not torch.isfinite(got[s, t, 1]).all()
        keep = torch.ones(seqs, T, heads, dtype=torch.bool, device="cuda")
        keep[s, t // 16 * 16:, 1] = False
        if where == 0:  # a query only meets its own token
            keep[s, t + 1:, 1] = True
            keep[s, t // 16 * 16:t, 1] = True
        assert torch.equal(got[keep], clean[keep])
