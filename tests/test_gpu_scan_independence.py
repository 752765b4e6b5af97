"""A sequence's outputs are the same bits in whatever company it is scanned: members of a population are compared with one another, on one rank
or several, in full waves and partial ones, so no choice of kernel, slices or CTAs may show."""
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


# four, two and one CTA per (sequence, head), for every number of 16-token blocks
@pytest.mark.parametrize("hidden,heads,seqs,groups", [(512, 1, 160, [(0, 1), (5, 30), (40, 60)]), (320, 2, 90, [(3, 2), (10, 35)]), (96, 1, 160, [(7, 3)])])
@pytest.mark.parametrize("T", [1, 16, 17, 40, 64, 77, 96, 100, 128])
def test_closed_form(H, hidden, heads, seqs, groups, T):
    bits_of_groups(H, hidden, heads, seqs, T, T % 2, 0, groups)


@pytest.mark.parametrize("where", [0, 1, 2, 3])  # on q, k, v, or in a fourth part of the same rows
@pytest.mark.parametrize("hidden,heads,seqs,T", [(512, 1, 3, 128), (512, 1, 30, 100), (512, 1, 70, 33), (320, 2, 20, 77), (96, 1, 160, 128)])
def test_closed_form_in_place(H, hidden, heads, seqs, T, where):
    """Four, two and one CTA per unit, with an output that lies where they still read, for both layouts of q, k and v."""
    import torch
    rng = np.random.default_rng(hidden + T)
    x = torch.from_numpy((rng.standard_normal((seqs * T, 4 * hidden)) * 0.3).astype(np.float32)).cuda()
    beta = torch.from_numpy(rng.standard_normal(seqs * T).astype(np.float32)).cuda()

    def scan(q, k, v, ld, out, ld_out):
        H.efla_scan(state=None, state_fp16=1, q=q, k=k, v=v, beta_raw=beta, ld_qkv=ld, ld_beta=1, beta_bias=-2.0, seqs_per_bias=1, hidden=hidden, heads=heads,
                    seqs=seqs, T=T, method=1, eps=1e-6, out=out, ld_out=ld_out, variant=0)
        assert H.device_error() == 0
        return out[:, :hidden].clone()

    apart = scan(x, x[:, hidden:], x[:, 2 * hidden:], 4 * hidden, torch.empty(seqs * T, hidden, device="cuda"), hidden)
    y = x.clone()
    rows = scan(y, y[:, hidden:], y[:, 2 * hidden:], 4 * hidden, y[:, where * hidden:], 4 * hidden)
    parts = [x[:, i * hidden:(i + 1) * hidden].contiguous() for i in range(4)]
    buffers = scan(*parts[:3], hidden, parts[where], hidden)
    assert torch.equal(rows, apart) and torch.equal(buffers, apart)


# wide rows (q | k | v | room), and rows of v alone that are narrower than two outputs, so that a row of y ends on the next row of v
@pytest.mark.parametrize("ld,shift", [(2048, 6), (2048, 64), (2048, 100), (2048, 128), (2048, 192), (2048, 256), (2048, 450), (2048, -8), (2048, -100), (576, 96), (640, 160)])
@pytest.mark.parametrize("seqs,T", [(1, 128), (1, 33), (200, 128)])
def test_closed_form_across_v(H, ld, shift, seqs, T):
    """One head of eight column tiles whose output lies on other columns of v."""
    import torch
    hidden = 512
    if ld < 2 * hidden and seqs > 1:
        pytest.skip("a sequence's last row lies on the next sequence")
    rng = np.random.default_rng(1000 + T + shift)
    qkv = [torch.from_numpy((rng.standard_normal((seqs * T + 1, ld)) * 0.3).astype(np.float32)).cuda() for _ in range(3)]
    beta = torch.from_numpy(rng.standard_normal(seqs * T).astype(np.float32)).cuda()

    def scan(v, out, ld_out):
        H.efla_scan(state=None, state_fp16=1, q=qkv[0], k=qkv[1], v=v, beta_raw=beta, ld_qkv=ld, ld_beta=1, beta_bias=-2.0, seqs_per_bias=1, hidden=hidden, heads=1, seqs=seqs, T=T,
                    method=1, eps=1e-6, out=out, ld_out=ld_out, variant=0)
        assert H.device_error() == 0

    first = 512 if ld >= 2 * hidden else 0  # column of v
    apart = torch.empty(seqs * T, hidden, device="cuda")
    scan(qkv[2][:, first:], apart, hidden)
    out = qkv[2].view(-1)[first + shift:]
    scan(qkv[2][:, first:], out, ld)
    assert torch.equal(torch.as_strided(out, (seqs * T, hidden), (ld, 1)), apart)


@pytest.mark.parametrize("hidden,heads,method", [(96, 1, 1), (512, 8, 1), (128, 4, 0)])
def test_other_scans(H, hidden, heads, method):
    """One CTA (128-token blocks) or one warp per unit, whatever their number."""
    bits_of_groups(H, hidden, heads, 40, 130, method, 0, [(0, 1), (11, 20)])


@pytest.mark.parametrize("T", [768, 769, 1024])
def test_long_closed_form(H, T):
    bits_of_groups(H, 96, 1, 34, T, 1, 0, [(0, 1), (2, 31)])


def test_losses_of_a_population_do_not_depend_on_the_wave():
    """Wide heads: 2, 6 and 18 members a wave take four, two and one CTA per (sequence, head)."""
    import torch
    from bitnet_nvfp4_b200 import population, synth
    out = []
    for wave in (2, 6, 18):
        cfg = population.Config(hidden=256, heads=1, layers=1, seq=40, batch=9, max_pairs=9, wave_members=wave)
        model = population.PopulationModel(cfg)
        model.set_weights(synth.init_weights(cfg))
        model.set_tokens(*synth.sample_batch(synth.zipf_corpus(1 << 14, 1.1, 123), 9, 40, 7))
        model.prepare_step(3, 1, 9)
        out.append(model.eval_pairs(0, 9))
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
