"""Closed form of whole sequences: values that are no numbers, and values of very different size. The recurrence is causal, so tokens before
such a value come out as without it, and what it makes NaN behind it is NaN here too."""
import numpy as np
import pytest

from test_gpu_scan_forms import H, exact_scan, make_qkv, run  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = [(512, 1, 2, 128), (96, 1, 170, 50), (320, 2, 40, 77), (96, 1, 2, 1), (512, 1, 3, 300), (192, 2, 2, 513)]


@pytest.mark.parametrize("method", [1, 0])
@pytest.mark.parametrize("hidden,heads,seqs,T", SHAPES)
@pytest.mark.parametrize("where", ["q", "k", "v", "beta"])
def test_tokens_before_a_value_that_is_no_number(H, hidden, heads, seqs, T, method, where):
    rng = np.random.default_rng(hidden + T)
    fc = (3 * hidden + 1 + 31) & ~31
    qkv = make_qkv(rng, seqs * T, hidden, fc, 0.3).reshape(seqs, T, fc)
    bb = np.full(seqs, -2.0, np.float32)
    clean = run(H, qkv.reshape(-1, fc), bb, 1, hidden, heads, seqs, T, method, 0)
    bad = qkv.copy()
    for s in range(seqs):
        for value in (np.nan, np.inf, -np.inf)[:1 + s % 3]:
            t = int(rng.integers(0, T)) if s % 4 else (0, T - 1)[s % 8 == 0]
            c = 3 * hidden if where == "beta" else "qkv".index(where) * hidden + int(rng.integers(0, hidden))
            bad[s, t, c] = value if where != "beta" or value != np.inf else np.nan
    got = run(H, bad.reshape(-1, fc), bb, 1, hidden, heads, seqs, T, method, 0)
    with np.errstate(all="ignore"):
        ref = exact_scan(bad, bb, hidden, heads, method)
    if where == "beta":  # (a logit of -infinity is a beta of zero, whose row of the recurrence is finite)
        assert np.isnan(got).any()
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert np.abs(got[ok] - ref[ok]).max(initial=0) <= 2e-5 * ((T + 127) // 128) * np.abs(clean).max()
    before = np.cumsum(~ok, axis=1) == 0
    if where != "beta":
        assert np.abs(got[before] - clean[before]).max(initial=0) <= 1e-6 * np.abs(clean).max()


@pytest.mark.parametrize("method", [1, 0])
@pytest.mark.parametrize("T", [60, 200])
def test_norms_that_overflow(H, T, method):
    """A finite k whose squared norm is infinite: alpha (or the scale of k) is zero and the token leaves the state alone, q comes out as zero."""
    rng = np.random.default_rng(T)
    hidden, fc, seqs = 96, 320, 2
    qkv = make_qkv(rng, seqs * T, hidden, fc, 0.3).reshape(seqs, T, fc)
    bb = np.full(seqs, -2.0, np.float32)
    without = qkv.copy()
    qkv[0, 7, hidden:2 * hidden] = 1e25
    qkv[1, T - 3, :hidden] = -1e30
    got = run(H, qkv.reshape(-1, fc), bb, 1, hidden, 1, seqs, T, method, 0)
    assert np.isfinite(got).all() and not got[1, T - 3].any()
    without[0, 7, hidden:2 * hidden] = 0.0  # (a zero key changes nothing either)
    ref = exact_scan(without, bb, hidden, 1, method)
    ref[1, T - 3] = 0.0
    assert np.abs(got - ref).max() <= 4e-5 * np.abs(ref).max()


@pytest.mark.parametrize("ratio", [1e2, 1e5, 1e7, 1e8])
@pytest.mark.parametrize("hidden,T", [(512, 128), (96, 40), (96, 200)])
def test_tokens_much_smaller_than_later_ones(H, hidden, T, ratio):
    """Rows of small values before large ones of their tile: off by no more than the form with fp16 states has them, relative to themselves."""
    rng = np.random.default_rng(int(ratio) + T)
    fc, seqs, half = (3 * hidden + 1 + 31) & ~31, 4, min(T, 128) // 2
    qkv = make_qkv(rng, seqs * T, hidden, fc, 0.3).reshape(seqs, T, fc)
    qkv[:, :half, 2 * hidden:3 * hidden] *= np.float32(1e-2)
    qkv[:, half:, 2 * hidden:3 * hidden] *= np.float32(1e-2 * ratio)
    if ratio > 1e7:  # (within fp16's range for the other form)
        qkv[:, :, 2 * hidden:3 * hidden] *= np.float32(0.1)
    bb = np.full(seqs, -2.0, np.float32)
    ref = exact_scan(qkv, bb, hidden, 1, 1)[:, :half]
    err = [np.abs(run(H, qkv.reshape(-1, fc), bb, 1, hidden, 1, seqs, T, 1, variant)[:, :half] - ref).max() / np.abs(ref).max() for variant in (0, 1)]
    assert err[0] <= max(err[1], 1e-6), err
