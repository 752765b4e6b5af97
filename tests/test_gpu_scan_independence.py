"""A sequence's outputs are the same bits in whatever company it is scanned: members of a population are compared with one another, on one rank
or several, in full waves and partial ones, so no choice of kernel, slices or clusters may show."""
import numpy as np
import pytest

from test_gpu_scan_forms import H, make_qkv, run  # noqa: F401

pytestmark = pytest.mark.gpu


def bits_of_groups(H, hidden, heads, seqs, T, method, variant, groups):
    rng = np.random.default_rng(hidden + T)
    fc = (3 * hidden + 1 + 31) & ~31
    qkv = make_qkv(rng, seqs * T, hidden, fc, 0.3).reshape(seqs, T, fc)
    bb = (rng.standard_normal(seqs) * 0.2 - 2.0).astype(np.float32)
    whole = run(H, qkv.reshape(-1, fc), bb, 1, hidden, heads, seqs, T, method, variant)
    for first, count in groups:
        part = run(H, qkv[first:first + count].reshape(-1, fc), bb[first:first + count], 1, hidden, heads, count, T, method, variant)
        assert np.array_equal(part, whole[first:first + count]), (first, count)


@pytest.mark.parametrize("hidden,heads,method", [(512, 1, 1), (1024, 2, 0), (320, 1, 1), (96, 1, 1), (1280, 1, 0)])
def test_per_token_kernel(H, hidden, heads, method):
    bits_of_groups(H, hidden, heads, 48, 5, method, 1, [(0, 1), (3, 8), (17, 19)])
