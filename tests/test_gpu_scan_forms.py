"""EFLA scan for head widths other than 64: the closed form of a whole sequence (zero state) and the
generic per-token kernel's column / row splits.

The closed form rounds nothing to fp16 between tokens, so it is held to the recurrence in float64. Its operands carry 22
significant bits (two fp16 terms) and sums accumulate in fp32: an element of G, X, P~ or y is a sum of at most 512 products
whose factors are off by 2^-22 each, rounded 512 times at 2^-24 relative to the running sum; rows are normalised, so errors are
relative to max |y| up to the growth of the triangular solve (entries of the inverse are at most 1 here). 2e-5 of max |y| leaves
a factor of about ten.
"""
import numpy as np
import pytest

import oracle_lib as orc

pytestmark = pytest.mark.gpu
SCAN_TOL = 2e-3  # fp16 state against fp16 state, as for the other scan kernels


@pytest.fixture(scope="module")
def H():
    import torch
    from bitnet_nvfp4_b200 import host
    assert torch.cuda.is_available()
    return host


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def make_qkv(rng, rows, hidden, fc, scale):
    qkv = np.zeros((rows, fc), np.float32)
    qkv[:, :3 * hidden] = (rng.standard_normal((rows, 3 * hidden)) * scale).astype(np.float32)
    qkv[:, 3 * hidden] = rng.standard_normal(rows).astype(np.float32)
    return qkv


def exact_scan(qkv, bb_seq, hidden, heads, method, eps=1e-6):
    """The recurrence in float64 without any rounding of the state."""
    seqs, T, _ = qkv.shape
    hd = hidden // heads
    x = qkv.astype(np.float64)
    q, k, v = (x[:, :, i * hidden:(i + 1) * hidden].reshape(seqs, T, heads, hd) for i in range(3))
    beta = 1.0 / (1.0 + np.exp(-(x[:, :, 3 * hidden] + bb_seq[:, None])))[:, :, None]
    q = q / np.sqrt((q ** 2).sum(-1, keepdims=True) + eps)
    lam = np.maximum((k ** 2).sum(-1), eps)
    if method == 0:
        alpha, k = beta * np.ones_like(lam), k / np.sqrt(lam + eps)[..., None]
    else:
        alpha = -np.expm1(-beta * lam) / (lam + eps)
    S = np.zeros((seqs, heads, hd, hd))
    y = np.empty((seqs, T, heads, hd))
    for t in range(T):
        diff = v[:, t] - np.einsum("shd,shdn->shn", k[:, t], S)
        S += (alpha[:, t, :, None] * k[:, t])[..., None] * diff[:, :, None, :]
        y[:, t] = np.einsum("shd,shdn->shn", q[:, t], S)
    return y.reshape(seqs, T, hidden)


def run(H, qkv, bb, per_bias, hidden, heads, seqs, T, method, variant, state=None):
    import torch
    qd = dev(qkv)
    fc = qkv.shape[1]
    out = torch.full((seqs * T, hidden), float("nan"), device="cuda")
    H.efla_scan(state=state, state_fp16=1, q=qd, k=qd[:, hidden:], v=qd[:, 2 * hidden:], beta_raw=qd[:, 3 * hidden:], ld_qkv=fc, ld_beta=fc,
                beta_bias_seq=dev(bb), seqs_per_bias=per_bias, hidden=hidden, heads=heads, seqs=seqs, T=T, method=method, eps=1e-6, out=out,
                ld_out=hidden, variant=variant)
    return out.cpu().numpy().reshape(seqs, T, hidden)


@pytest.mark.parametrize("scale", [0.3, 1000.0, 1e-3])   # 1000: k, q, v far outside fp16's comfortable range; 1e-3: lambda near eps
@pytest.mark.parametrize("hidden,heads,seqs,T,method", [
    (512, 1, 3, 128, 1), (512, 1, 2, 100, 0), (256, 2, 3, 33, 1), (96, 1, 2, 17, 1), (320, 2, 2, 113, 0), (96, 1, 5, 1, 1), (256, 2, 2, 16, 1),
    (512, 1, 2, 47, 1),
    (512, 1, 40, 33, 1), (192, 2, 30, 20, 0), (96, 1, 160, 18, 1), (320, 1, 150, 16, 1)])   # two CTAs per unit; one
def test_closed_form_matches_the_exact_recurrence(H, hidden, heads, seqs, T, method, scale):
    rng = np.random.default_rng(hidden + T + method)
    fc = (3 * hidden + 1 + 31) & ~31
    qkv = make_qkv(rng, seqs * T, hidden, fc, scale)
    bb = (rng.standard_normal((seqs + 1) // 2) * 0.2 - 2.0).astype(np.float32)
    bb_seq = np.repeat(bb, 2)[:seqs]
    got = run(H, qkv, bb, 2, hidden, heads, seqs, T, method, 0)
    ref = exact_scan(qkv.reshape(seqs, T, fc), bb_seq, hidden, heads, method)
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("hidden,heads,seqs,T,method", [(96, 1, 3, 20, 1), (160, 1, 2, 9, 1), (1024, 1, 2, 5, 1), (256, 8, 4, 12, 0), (1280, 1, 1, 3, 1),
                                                        (512, 2, 3, 150, 1), (384, 1, 2, 140, 0), (512, 1, 3, 12, 1), (320, 1, 2, 9, 0), (512, 1, 20, 5, 1), (128, 4, 3, 33, 1), (32, 1, 5, 1, 1), (96, 3, 7, 130, 0)])
def test_generic_kernel_splits_match_the_oracle(H, hidden, heads, seqs, T, method):
    """Every split of the generic kernel (piece counts and rows per thread), and AUTO beyond 128 tokens."""
    rng = np.random.default_rng(hidden * 7 + T)
    fc = (3 * hidden + 1 + 31) & ~31
    qkv = make_qkv(rng, seqs * T, hidden, fc, 0.3)
    bb = (rng.standard_normal(seqs) * 0.2 - 2.0).astype(np.float32)
    got = run(H, qkv, bb, 1, hidden, heads, seqs, T, method, 1 if T <= 128 else 0)
    ref = orc.efla_scan(qkv.reshape(seqs, T, fc), bb, hidden, heads, method)
    assert np.abs(got - ref).max() <= SCAN_TOL * np.abs(ref).max()


@pytest.mark.parametrize("offset", [0, 1])  # a state that is not 16-byte aligned travels element by element
@pytest.mark.parametrize("fp16", [1, 0])
@pytest.mark.parametrize("hidden", [96, 32])
def test_generic_kernel_carries_the_state(H, hidden, fp16, offset):
    """Two calls of T1 and T2 tokens with the state in HBM between them = one call of T1 + T2 tokens, bit for bit."""
    import torch
    rng = np.random.default_rng(5)
    seqs, T1, T2 = 3, 4, 3
    fc = 320
    qkv = make_qkv(rng, seqs * (T1 + T2), hidden, fc, 0.4).reshape(seqs, T1 + T2, fc)
    bb = np.full(seqs, -2.0, np.float32)
    n = seqs * hidden * hidden

    def call(x, store, T):
        qd = dev(x.reshape(-1, fc))
        out = torch.empty((seqs * T, hidden), device="cuda")
        H.efla_scan(state=store[offset:], state_fp16=fp16, q=qd, k=qd[:, hidden:], v=qd[:, 2 * hidden:], beta_raw=qd[:, 3 * hidden:], ld_qkv=fc, ld_beta=fc,
                    beta_bias_seq=dev(bb), seqs_per_bias=1, hidden=hidden, heads=1, seqs=seqs, T=T, method=1, eps=1e-6, out=out, ld_out=hidden, variant=0)
        return out.cpu().numpy().reshape(seqs, T, hidden)

    dt = torch.float16 if fp16 else torch.float32
    one, two = torch.zeros(n + 1, dtype=dt, device="cuda"), torch.zeros(n + 1, dtype=dt, device="cuda")
    whole = call(qkv, one, T1 + T2)
    parts = np.concatenate([call(qkv[:, :T1], two, T1), call(qkv[:, T1:], two, T2)], axis=1)
    assert np.array_equal(whole, parts)
    assert torch.equal(one, two)


@pytest.mark.parametrize("scale", [0.3, 1000.0, 1e-3])
@pytest.mark.parametrize("hidden,heads,seqs,T,method", [
    (512, 1, 2, 129, 1), (512, 1, 3, 322, 0), (96, 1, 2, 256, 1), (320, 2, 2, 257, 1), (128, 1, 150, 140, 0), (160, 1, 1, 768, 1),
    (96, 1, 32, 1024, 1), (96, 1, 2, 1024, 0)])
def test_closed_form_of_long_sequences(H, hidden, heads, seqs, T, method, scale):
    """More than one block of 128 tokens: one token in the last block, full blocks, more units than SMs, the longest of few and of many
    units. Every block product adds the error that the one-block form is allowed, so the bound grows with the number of blocks."""
    rng = np.random.default_rng(hidden + T + method)
    fc = (3 * hidden + 1 + 31) & ~31
    qkv = make_qkv(rng, seqs * T, hidden, fc, scale)
    bb = (rng.standard_normal((seqs + 1) // 2) * 0.2 - 2.0).astype(np.float32)
    bb_seq = np.repeat(bb, 2)[:seqs]
    got = run(H, qkv, bb, 2, hidden, heads, seqs, T, method, 0)
    ref = exact_scan(qkv.reshape(seqs, T, fc), bb_seq, hidden, heads, method)
    assert np.abs(got - ref).max() <= 2e-5 * ((T + 127) // 128) * np.abs(ref).max()


@pytest.mark.parametrize("on,shift", [("q", 0), ("k", 0), ("v", 0), ("v", 8), ("apart", 0)])
@pytest.mark.parametrize("hidden,seqs,T", [(96, 1, 150), (512, 300, 133), (1024, 40, 130)])
def test_long_sequence_into_its_own_inputs(H, hidden, seqs, T, on, shift):
    """An output that lies on q, k or v keeps the per-token kernel. The slices of a head (more CTAs than fit the device here) read whole rows
    of q and k, so they must not see one another's outputs: the same bits as into a buffer of its own."""
    import torch
    rng = np.random.default_rng(3)
    fc = 4 * hidden + 32
    qkv = make_qkv(rng, seqs * T, hidden, fc, 0.4)
    beta = dev(qkv[:, 3 * hidden])

    def scan(qd, out, ld):
        H.efla_scan(state=None, state_fp16=1, q=qd, k=qd[:, hidden:], v=qd[:, 2 * hidden:], beta_raw=beta, ld_qkv=fc, ld_beta=1, beta_bias=-2.0, hidden=hidden, heads=1,
                    seqs=seqs, T=T, method=1, eps=1e-6, out=out, ld_out=ld, variant=1)

    want = torch.empty(seqs * T, hidden, device="cuda")
    scan(dev(qkv), want, hidden)
    qd = dev(qkv)
    col = {"q": 0, "k": hidden, "v": 2 * hidden, "apart": 3 * hidden + 32}[on] + shift
    scan(qd, qd[:, col:], fc)
    assert torch.equal(qd[:, col:col + hidden], want)
    assert torch.equal(torch.cat([qd[:, :col], qd[:, col + hidden:]], 1), torch.cat([dev(qkv)[:, :col], dev(qkv)[:, col + hidden:]], 1))


def test_long_sequence_into_its_own_queries(H):
    """An output that overlays q keeps the per-token kernel."""
    import torch
    rng = np.random.default_rng(3)
    hidden, T, fc = 96, 150, 320
    qkv = make_qkv(rng, T, hidden, fc, 0.4)
    bb = np.full(1, -2.0, np.float32)
    ref = run(H, qkv, bb, 1, hidden, 1, 1, T, 1, 0)
    qd = dev(qkv)
    H.efla_scan(state=None, state_fp16=1, q=qd, k=qd[:, hidden:], v=qd[:, 2 * hidden:], beta_raw=dev(qkv[:, 3 * hidden]), ld_qkv=fc, ld_beta=1,
                beta_bias_seq=dev(bb), seqs_per_bias=1, hidden=hidden, heads=1, seqs=1, T=T, method=1, eps=1e-6, out=qd, ld_out=fc, variant=0)
    assert np.abs(qd[:, :hidden].cpu().numpy() - ref[0]).max() <= SCAN_TOL * np.abs(ref).max()
