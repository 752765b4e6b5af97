"""The mean loss of a member is one sum in one order, whatever the grid that forms it: members that rank against one another must not
change places with the number of blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab,batch,seq", [(256, 4, 16), (256, 31, 67), (256, 32, 64), (256, 32, 128), (256, 33, 131), (256, 32, 256), (250, 32, 128)])
def test_loss_of_a_model_equals_the_entry_point_bit_for_bit(vocab, batch, seq):
    """Zero head weights: the logits are zero, the row losses those of the bias, and only their summation is left."""
    import torch
    from bitnet_nvfp4_b200 import host, population, synth
    cfg = population.Config(vocab=vocab, hidden=128, layers=1, heads=2, seq=seq, batch=batch, max_pairs=1)
    rng = np.random.default_rng(batch * seq)
    w = synth.init_weights(cfg)
    w["head"] = np.zeros_like(w["head"])
    w["head_bias"] = rng.normal(size=vocab).astype(np.float32)
    tok, tgt = (rng.integers(0, vocab, (batch, seq)).astype(np.uint8) for _ in range(2))
    model = population.PopulationModel(cfg)
    model.set_weights(w)
    model.set_tokens(tok, tgt)
    logits = torch.zeros(batch * seq, vocab, device="cuda")
    want = host.cross_entropy_population(logits, vocab, torch.from_numpy(w["head_bias"]).cuda(), None, 0.0, torch.from_numpy(tgt).cuda(), vocab, 1, batch * seq)
    assert torch.equal(model.eval_base(), want)
    # ... and the entry point adds chains of rows w, w + 8, .. inside sixteen groups, the chains in order, the groups in double
    bias = torch.from_numpy(w["head_bias"]).cuda()
    row_of = np.array([host.cross_entropy_population(logits, vocab, bias, None, 0.0, torch.tensor([y], dtype=torch.uint8, device="cuda"), vocab, 1, 1).item()
                       for y in range(vocab)], np.float32)
    rows, per, total = row_of[tgt.ravel()], -(-batch * seq // 16), 0.0
    for g in range(16):
        group = np.float32(0)
        for c in range(8):
            chain = np.float32(0)
            for x in rows[g * per:(g + 1) * per][c::8]:
                chain += x
            group += chain
        total += float(group)
    assert np.float32(total / (batch * seq)) == want.item()


def test_losses_do_not_depend_on_the_wave():
    """Rows enough for shared groups, in waves small and large enough for both forms of the grid."""
    import torch
    from bitnet_nvfp4_b200 import population, synth
    pairs, out = 24, []
    for wave in (2, 8, 48):
        cfg = population.Config(hidden=128, layers=1, heads=2, seq=128, batch=32, max_pairs=pairs, wave_members=wave)
        model = population.PopulationModel(cfg)
        model.set_weights(synth.init_weights(cfg))
        model.set_tokens(*synth.sample_batch(synth.zipf_corpus(1 << 14, 1.1, 123), 32, 128, 7))
        model.prepare_step(3, 1, pairs)
        out.append(model.eval_pairs(0, pairs))
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
