"""The step's device-side path: fitness shaping, noise sums from the noise tables, the update that renews the NVFP4 copies in the
same pass, single-member validation, and a model narrower than its vocabulary. Integer and shaping results are compared bit for bit."""
import numpy as np
import pytest

import oracle_lib as orc

pytestmark = pytest.mark.gpu


def make(seed=3, **kw):
    import torch
    from bitnet_nvfp4_b200 import population, synth
    assert torch.cuda.is_available()
    cfg = population.Config(**kw)
    w = synth.init_weights(cfg)
    tok, tgt = (np.ascontiguousarray(np.minimum(x, cfg.vocab - 1)) for x in synth.sample_batch(synth.zipf_corpus(1 << 14, 1.1, 123), cfg.batch, cfg.seq, seed))
    model = population.PopulationModel(cfg)
    model.set_weights(w)
    model.set_tokens(tok, tgt)
    return cfg, w, tok, tgt, model


def oracle_loss(cfg, w, tok, tgt):
    ocfg = {k: getattr(cfg, k) for k in "vocab hidden layers mlp_mult seq batch heads rank sigma_shift use_clt clt_k method act_scale "
                                        "mlp_act_scale ln_scale residual_scale mlp_residual_scale eps".split()}
    return orc.OracleModel(ocfg, w).forward(tok, tgt, 0, 0)


def state(model):
    w = model.get_weights()
    shadow, ema = model.get_optimizer_state()
    return [w[n] for n in sorted(w)] + [shadow, ema]


SMALL = dict(hidden=128, layers=1, seq=16, batch=4, heads=2)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("pairs", [1, 2, 37, 1030])  # 1030: more than one element per thread of the shaping kernel
def test_device_shaping_equals_the_host_function(mode, pairs):
    """marks asks for the composed step, whose shaping is the host function; without it the step shapes on the device."""
    from bitnet_nvfp4_b200 import population
    results = []
    for marks in (None, {}):
        _, _, _, _, m = make(max_pairs=pairs, **SMALL)
        losses = [population.es_step(m, 5, e, pairs, fitness_mode=mode, fitness_clip=1.5, marks=marks).cpu().numpy() for e in range(2)]
        results.append(losses + state(m))
    for a, b in zip(*results):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("pairs", [3, 17, 40])
def test_noise_sums_from_tables_equal_the_hashed_ones(pairs):
    """A process that evaluated every pair finds the vectors' noise in memory; one that evaluated none hashes it."""
    import torch
    w = torch.linspace(-0.5, 0.5, pairs, device="cuda")
    w[pairs // 2] = 0.0
    out = []
    for count in (pairs, 0):
        _, _, _, _, m = make(max_pairs=pairs, **SMALL)
        m.prepare_step_range(9, 1, pairs, 0, count)
        m.update(w, lr=0.7, thresh=0.001)
        out.append(state(m))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("use_clt,clt_k", [(1, 127), (1, 128), (1, 20000), (0, 20000)])
def test_noise_sums_of_draws_that_exceed_a_byte(use_clt, clt_k):
    """20000 ternary draws sum to some 115: one in four sums does not fit the byte that the evaluation reads, and the update takes the sum itself."""
    import torch
    w = torch.tensor([0.5, -0.25, 0.125], device="cuda")
    out = []
    for count in (3, 0):
        _, _, _, _, m = make(max_pairs=3, use_clt=use_clt, clt_k=clt_k, **SMALL)
        m.prepare_step_range(9, 1, 3, 0, count)
        m.update(w, lr=0.7, thresh=0.001)
        out.append(state(m))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kw", [dict(SMALL), dict(hidden=192, layers=2, mlp_mult=3, seq=9, batch=3, heads=3, rank=2), dict(hidden=64, layers=1, seq=32, batch=9, heads=1, rank=4)])
def test_validation_after_an_update_matches_the_oracle(kw):
    """The update renews the NVFP4 copies of the weights itself: the next forward (one unperturbed member) is the oracle's at the updated
    weights. The last case is narrower than its vocabulary of 256."""
    from bitnet_nvfp4_b200 import host, population
    cfg, w, tok, tgt, m = make(max_pairs=6, **kw)
    assert abs(m.eval_base().item() - oracle_loss(cfg, w, tok, tgt)) <= 1e-4 * 6
    population.es_step(m, 1, 0, 6, lr=1.5, thresh=0.004)
    after = m.get_weights()
    assert any(not np.array_equal(after[n], w[n]) for n in ("wq", "ff1", "head"))
    ref = oracle_loss(cfg, after, tok, tgt)
    assert abs(m.eval_base().item() - ref) <= 1e-4 * abs(ref)
    assert host.device_error() == 0


@pytest.mark.parametrize("kw", [
    dict(hidden=128, layers=2, seq=64, batch=6, heads=2, max_pairs=5),                     # several pairs per wave, tokens de-duplicated
    dict(hidden=192, layers=1, mlp_mult=3, seq=32, batch=4, heads=3, max_pairs=3, vocab=200),  # vocabulary that is no multiple of a tile, K remainder of 64
    dict(hidden=128, layers=1, seq=32, batch=12, heads=1, max_pairs=2, sigma_shift=6),     # sigma too small for the folded form
])
def test_dense_noise_in_one_product(kw):
    """rank 0: base weights and each member's noise operand in one accumulation (sigma >= 2^-4), product by product below: member losses
    against the oracle's dense forward, and independence of the wave."""
    from bitnet_nvfp4_b200 import host
    cfg, w, tok, tgt, m = make(rank=0, **kw)
    pairs = cfg.max_pairs
    m.prepare_step(1, 3, pairs)
    losses = m.eval_pairs(0, pairs).cpu().numpy()
    assert host.device_error() == 0
    ocfg = {k: getattr(cfg, k) for k in "vocab hidden layers mlp_mult seq batch heads rank sigma_shift use_clt clt_k method act_scale "
                                        "mlp_act_scale ln_scale residual_scale mlp_residual_scale eps".split()}
    om = orc.OracleModel(ocfg, w)
    for p in range(pairs):
        for s, anti in enumerate((1, -1)):
            ref = om.forward(tok, tgt, orc.mix(1, orc.mix(3, p)), anti)
            assert abs(losses[2 * p + s] - ref) <= 1e-4 * abs(ref), (p, anti)
    assert np.array_equal(m.eval_pairs(1, pairs - 1).cpu().numpy(), losses[2:])


@pytest.mark.parametrize("native", [True, False])
def test_a_pinned_batch_may_be_refilled_after_the_step(native):
    """The device is busy when the batch is set, so its copy is still queued when the host gets to the next one."""
    import torch
    from bitnet_nvfp4_b200 import population, synth
    busy = torch.randn(8192, 8192, device="cuda", dtype=torch.bfloat16)
    batches = [synth.sample_batch(synth.zipf_corpus(1 << 14, 1.1, 5), SMALL["batch"], SMALL["seq"], 20 + e) for e in range(4)]
    results = []
    for refill in (False, True):
        _, _, _, _, m = make(max_pairs=6, **SMALL)
        tok, tgt = (torch.empty(SMALL["batch"], SMALL["seq"], dtype=torch.uint8, pin_memory=True) for _ in range(2))
        losses = []
        for e, (a, b) in enumerate(batches):
            tok.copy_(torch.from_numpy(a))
            tgt.copy_(torch.from_numpy(b))
            if refill:
                for _ in range(40):
                    torch.mm(busy, busy)
            m.set_tokens(tok, tgt)
            losses.append((population.es_step_native if native else population.es_step)(m, 5, e, 6))
            if not refill:
                torch.cuda.synchronize()
        results.append([x.cpu().numpy() for x in losses] + state(m))
    for a, b in zip(*results):
        assert np.array_equal(a, b)


def test_weights_go_into_the_callers_arrays_and_nowhere_else():
    """Host arrays that lie like the device's (1024-byte steps) with a caller's data between them, and the one-copy form."""
    import ctypes as C

    from bitnet_nvfp4_b200 import lib, population
    cfg, w, _, _, m = make(max_pairs=1, **SMALL)
    layout, at = [], 0
    for n, shape in cfg.weight_shapes().items():
        nbytes = int(np.prod(shape)) * (4 if n in ("head_bias", "beta_bias", "pos") else 1)
        layout.append((n, shape, at, nbytes))
        at += -(-nbytes // 1024) * 1024
    assert any(nbytes % 1024 for _, _, _, nbytes in layout[:-1])
    block = np.full(at, 0xA5, np.uint8)
    lib.check(m.lib.bnf4_model_get_weights(m.h, C.byref(population.ModelWeights(*[block.ctypes.data + a for _, _, a, _ in layout]))))
    one = np.zeros(at, np.uint8)
    lib.check(m.lib.bnf4_model_get_weights_block(m.h, one.ctypes.data, at))
    mine = np.ones(at, bool)
    for n, shape, a, nbytes in layout:
        want = np.frombuffer(np.ascontiguousarray(w[n]).tobytes(), np.uint8)
        assert np.array_equal(block[a:a + nbytes], want) and np.array_equal(one[a:a + nbytes], want) and np.array_equal(m.get_weights()[n], w[n])
        mine[a:a + nbytes] = False
    assert (block[mine] == 0xA5).all()
    with pytest.raises(lib.Bnf4Error):
        lib.check(m.lib.bnf4_model_get_weights_block(m.h, one.ctypes.data, at - 1024))


def test_kept_weights_do_not_pile_up_page_locked_memory(monkeypatch):
    import gc

    import torch
    from bitnet_nvfp4_b200 import population
    _, w, _, _, m = make(max_pairs=1, **SMALL)
    gc.collect()
    size = sum(-(-a.nbytes // 1024) * 1024 for a in m.get_weights().values())
    gc.collect()
    assert population._pinned_bytes == 0
    monkeypatch.setattr(population, "_PINNED_TOTAL", 3 * size)
    kept = [m.get_weights() for _ in range(5)]
    assert population._pinned_bytes == 3 * size
    assert [torch.from_numpy(k["emb"]).is_pinned() for k in kept] == [True] * 3 + [False] * 2
    assert all(np.array_equal(k[n], w[n]) for k in kept for n in w)
    one = kept[0]["head"]
    del kept
    gc.collect()
    assert population._pinned_bytes == size
    del one
    gc.collect()
    assert population._pinned_bytes == 0
