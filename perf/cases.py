"""The work whose speed matters to users of this package, as cases that can be timed one by one.

A case is a dict of plain values with a "kind":

  epoch     one epoch of training as the epoch loop runs it (trainer.train): the epoch's batch from pinned host memory, the ES
            step (per-pair noise, evaluation of every antithetic pair, fitness shaping, update, re-quantisation) and the loss of
            the updated model on that batch; with "keep", also the read-back of the weights that a program does when it keeps them.
  validate  the loss of the unperturbed model on a batch (the validation pass of the epoch loop).
  token     one token step of the reference driver's own loop through the reference-shaped entry points (M = batch rows per GEMM,
            state of every layer in device memory): what a program that links the library in place of the reference's kernels runs.
  perturbed activations quantised on the fly and multiplied with ternary weights plus a rank-r term per member, all members in one call.
  gemm      the block-scaled GEMM alone, on operands that are quantised already.
  scan      the EFLA / DeltaNet recurrence alone over whole sequences.
  update    noise sum, RMS normalisation and shadow / ternary update of one weight matrix.

Sizes: the default model, the smoke-test model, the scaled-up stress widths, the one-head and dense-noise forms of the reference,
the single perturbed GEMM (4 members, M 4096, K = N 512) and the GEMM sweep up to M 16384, K = N 4096.
"""
import math

import numpy as np
import torch

from bitnet_nvfp4_b200 import host, population, synth

VOCAB = 256
EPILOGUES = ("f32", "f16", "add_i8", "gelu_i8", "gelu_fp4")


def _epoch(name, hidden, heads, layers, mlp_mult, seq, batch, rank, pairs, method=1, keep=False):
    return {"name": name, "kind": "epoch", "hidden": hidden, "heads": heads, "layers": layers, "mlp_mult": mlp_mult, "seq": seq,
            "batch": batch, "rank": rank, "pairs": pairs, "method": method, "keep": keep}


def listed():
    return [
        # the smallest training run: the smoke-test model with a handful of pairs, where launches and host work decide
        _epoch("epoch smoke", 128, 2, 2, 2, 32, 8, 1, 4, keep=True),
        # the default model at its full population of 2048: the workload the package is built for
        _epoch("epoch default", 512, 8, 4, 2, 128, 32, 1, 1024, keep=True),
        # sizes that are multiples of nothing in particular, DeltaNet instead of EFLA, rank 2, a population that fills no wave
        _epoch("epoch ragged", 320, 5, 3, 3, 100, 12, 2, 37, method=0, keep=True),
        # the stress widths (hidden 2048, MLP 8192, 32 heads, sequences of 512, rank 4) with three of their layers; an epoch whose
        # weights stay on the GPU, as most do (their read-back would take as long as the step)
        _epoch("epoch wide", 2048, 32, 3, 4, 512, 16, 4, 16),
        # the reference's own head layout (one head as wide as the model) at the default sizes, with low-rank perturbations
        _epoch("epoch one head", 512, 1, 4, 2, 128, 32, 1, 16, keep=True),
        # the reference's own form throughout: one head and dense noise matrices, a second GEMM per projection
        _epoch("epoch dense", 512, 1, 4, 2, 128, 32, 0, 4, keep=True),
        # validation between two epochs: one forward of the unperturbed default model, a latency
        {"name": "validate default", "kind": "validate", "hidden": 512, "heads": 8, "layers": 4, "mlp_mult": 2, "seq": 128, "batch": 32, "method": 1},
        # the reference's token loop at its default sizes, perturbed by its dense noise: many small calls
        {"name": "token default", "kind": "token", "hidden": 512, "layers": 4, "mlp_mult": 2, "batch": 32, "noisy": True},
        # the perturbed GEMM with its quantiser, four members of batch 32 x seq 128
        {"name": "perturbed 4 x 4096", "kind": "perturbed", "members": 4, "rows": 4096, "k": 512, "n": 512, "rank": 1},
        # the largest point of the GEMM sweep: the tensor cores' case
        {"name": "gemm 16384 x 4096", "kind": "gemm", "m": 16384, "n": 4096, "k": 4096, "rank": 4, "epilogue": "f32"},
        # the scan in its exact form (fp16 state after every token, as the reference rounds) over the sequences of 32 default members
        {"name": "scan exact", "kind": "scan", "seqs": 1024, "seq": 128, "heads": 8, "variant": "per_token", "half": False, "method": 1},
        # the reference driver's update of one default ff matrix from dense noise of a full population
        {"name": "update ff", "kind": "update", "form": "dense", "rows": 1024, "cols": 512, "pairs": 1024, "rank": 0},
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _model_shape(rng):
    hidden = 64 * _log(rng, 2, 32)
    layout = rng.random()
    heads = hidden // 64                                     # heads of 64: the benchmark's layout
    if layout > 0.85 and hidden <= 512:
        heads = 1                                            # the reference's
    elif layout > 0.75:
        heads = hidden // 32                                 # smaller heads
    return {"hidden": hidden, "heads": heads, "layers": rng.randint(1, 6), "mlp_mult": rng.randint(1, 4), "seq": _log(rng, 16, 512),
            "batch": _log(rng, 2, 32), "method": 1 if rng.random() < 0.75 else 0}


def _load(c):
    """Rough cost of an epoch: its operations, with the recurrence of other head sizes than 64 counted at what CUDA cores make of it."""
    h, hd = c["hidden"], c["hidden"] // c["heads"]
    rows = (2 * c["pairs"] + 2) * c["batch"] * c["seq"]
    scan = 6.0 * h * hd * (1 if hd == 64 else 250)
    per_row = c["layers"] * (2.0 * h * h * (3 + 2 * c["mlp_mult"]) + scan) + 2.0 * VOCAB * h
    dense = 30.0 * c["pairs"] * _params(c) * (60 if c["rank"] == 0 else 0)
    return rows * per_row + dense


def draw(rng):
    u = rng.random()
    if u < 0.55:
        c = {"kind": "epoch", **_model_shape(rng)}
        c["rank"] = rng.choice((1, 1, 2, 3, 4, 4))
        c["pairs"] = _log(rng, 2, 1024)
        if rng.random() < 0.12 and (c["batch"] * c["seq"]) % 128 == 0:
            c["rank"], c["pairs"] = 0, min(c["pairs"], 8)
        top = max(_load(e) for e in listed() if e["kind"] == "epoch")
        while _load(c) > top and c["pairs"] > 2:
            c["pairs"] = max(2, c["pairs"] * 2 // 3)
        while _load(c) > top:
            c["layers"], c["seq"] = max(1, c["layers"] - 1), max(16, c["seq"] // 2)
        if c["rank"] == 0 and (c["batch"] * c["seq"]) % 128 != 0:
            c["rank"] = 1
        c["keep"] = rng.random() < 0.6 and _params(c) < (8 << 20)
        return c
    if u < 0.62:
        return {"kind": "validate", **_model_shape(rng)}
    if u < 0.70:
        return {"kind": "token", "hidden": 128 * _log(rng, 1, 8), "layers": rng.randint(1, 6), "mlp_mult": rng.randint(1, 4),
                "batch": _log(rng, 4, 128), "noisy": rng.random() < 0.7}
    if u < 0.78:
        return {"kind": "perturbed", "members": _log(rng, 1, 16), "rows": _log(rng, 128, 4096), "k": 64 * _log(rng, 2, 32), "n": 64 * _log(rng, 2, 32),
                "rank": rng.randint(0, 4)}
    if u < 0.88:
        n = 64 * _log(rng, 1, 64)
        epilogue = rng.choice(EPILOGUES)
        if epilogue in ("f32", "f16") and rng.random() < 0.3:
            n += 1                                           # the stacked q | k | v | beta projection has such a width
        return {"kind": "gemm", "m": _log(rng, 64, 16384), "n": n, "k": 64 * _log(rng, 1, 64), "rank": rng.choice((0, 1, 1, 2, 4)), "epilogue": epilogue}
    if u < 0.94:
        heads, seq = _log(rng, 1, 16), _log(rng, 16, 512)
        variant = rng.choice(("auto", "per_token"))
        return {"kind": "scan", "seqs": _log(rng, 4, max(5, (1024 * 128 * 8) // (heads * seq))), "seq": seq, "heads": heads, "variant": variant,
                "half": variant == "auto" and rng.random() < 0.5, "method": 1 if rng.random() < 0.75 else 0}
    form = rng.choice(("dense", "lowrank"))
    rows, cols = _log(rng, 1, 2048), 16 * _log(rng, 2, 128)
    pairs = _log(rng, 2, max(3, min(1024, (1024 * 512 * 1024) // (rows * cols))))
    return {"kind": "update", "form": form, "rows": rows, "cols": cols, "pairs": pairs, "rank": rng.randint(1, 4) if form == "lowrank" else 0}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _ternary(g, *shape):
    return torch.randint(-1, 2, shape, device="cuda", generator=g, dtype=torch.int8)


def _clt(g, *shape):
    """Integer noise with the distribution of a sum of four ternary draws."""
    return sum(_ternary(g, *shape) for _ in range(4))


def _activations(g, *shape):
    """int8 activations as the abs-mean norm leaves them: most within a few units of zero, some far out."""
    return torch.clamp(torch.round(torch.randn(*shape, device="cuda", generator=g) * 40), -127, 127).to(torch.int8)


def _prepare_model(case, seed):
    cfg = population.Config(hidden=case["hidden"], heads=case["heads"], layers=case["layers"], mlp_mult=case["mlp_mult"], seq=case["seq"],
                            batch=case["batch"], method=case["method"], rank=case.get("rank", 1), max_pairs=case.get("pairs", 1))
    g = _gen(seed)
    w = {name: _ternary(g, *shape).cpu().numpy() for name, shape in cfg.weight_shapes().items() if name not in ("head_bias", "beta_bias", "pos")}
    w["head_bias"] = np.zeros(VOCAB, np.float32)
    w["beta_bias"] = np.full(cfg.layers, -2.0, np.float32)
    w["pos"] = ((torch.rand(cfg.seq, cfg.hidden, device="cuda", generator=g) - 0.5) * 0.04).cpu().numpy()
    model = population.PopulationModel(cfg)
    model.set_weights(w)
    tokens, targets = synth.sample_batch(synth.zipf_corpus(1 << 16, seed=seed), cfg.batch, cfg.seq, seed + 1)
    return {"model": model, "tokens": torch.from_numpy(tokens).pin_memory(), "targets": torch.from_numpy(targets).pin_memory(), "seed": seed,
            "epoch": 0, "pairs": case.get("pairs", 0), "keep": case.get("keep", False)}


def _prepare_token(case, seed):
    H, F, B, L = case["hidden"], case["hidden"] * case["mlp_mult"], case["batch"], case["layers"]
    g = _gen(seed)
    s_h = 1.0 / math.sqrt(H)
    fc = 3 * H + 32                                          # q | k | v | beta, padded as the reference pads it

    def quant(w):
        return host.nvfp4_quantize_b(w)

    def stacked(draw_):
        return host.nvfp4_quantize_wqkv_fused(draw_(g, H, H), draw_(g, H, H), draw_(g, H, H), draw_(g, 1, H), H, fc, s_h)

    def matrices(draw_):
        return {"win": quant(draw_(g, H, H)), "head": quant(draw_(g, VOCAB, H)),
                "layers": [{"qkv": stacked(draw_), "ff1": quant(draw_(g, F, H)), "ff2": quant(draw_(g, H, F))} for _ in range(L)]}

    st = {"case": case, "w": matrices(_ternary), "e": matrices(_clt) if case["noisy"] else None, "emb": _ternary(g, VOCAB, H),
          "emb_noise": _clt(g, VOCAB, H) if case["noisy"] else None, "bias": torch.zeros(VOCAB, device="cuda"),
          "pos": (torch.rand(H, device="cuda", generator=g) - 0.5) * 0.04,
          "S": [torch.zeros(B, H, H, dtype=torch.float16, device="cuda") for _ in range(L)], "loss": torch.zeros(1, device="cuda")}
    corpus = synth.zipf_corpus(1 << 14, seed=seed)
    st["tokens"], st["targets"] = (torch.from_numpy(x).cuda() for x in synth.sample_batch(corpus, B, 1, seed + 1))
    return st


def _prepare_perturbed(case, seed):
    members, rows, k, n, rank = case["members"], case["rows"], case["k"], case["n"], case["rank"]
    g, m = _gen(seed), members * rows
    pairs = (members + 1) // 2
    b, sfb = host.nvfp4_quantize_b(_ternary(g, n, k))
    st = {"case": case, "x": torch.randn(m, k, device="cuda", generator=g) * 0.8, "b": b, "sfb": sfb,
          "codes": torch.zeros(host.matrix_bytes(m, k), dtype=torch.uint8, device="cuda"),
          "sf": torch.zeros(host.sf_bytes(m, k), dtype=torch.uint8, device="cuda"), "d": torch.empty(m, n, device="cuda")}
    if rank > 0:
        st["A"], st["Bt"] = _clt(g, pairs, n, rank), _clt(g, pairs, rank, k)
        st["t"] = torch.zeros(m, rank, dtype=torch.int32, device="cuda")
    return st


def _prepare_gemm(case, seed):
    m, n, k, rank, epi = case["m"], case["n"], case["k"], case["rank"], case["epilogue"]
    g = _gen(seed)
    rpm = min(4096, m)                                       # rows per member
    pairs = (m + 2 * rpm - 1) // (2 * rpm)
    a, sfa = host.nvfp4_quantize_a(_activations(g, m, k))
    b, sfb = host.nvfp4_quantize_b(_ternary(g, n, k))
    kw = dict(a=a, b=b, sfa=sfa, sfb=sfb, m=m, n=n, k=k, alpha=1.0 / math.sqrt(k))
    if rank > 0:
        kw.update(rank=rank, rows_per_member=rpm, lora_t=torch.randint(-1000, 1000, (m, rank), device="cuda", generator=g, dtype=torch.int32),
                  t_stride=rank, lora_A=_clt(g, pairs, n, rank), lora_A_pair_stride=n * rank, lora_scale=0.125 * host.c_rank(rank) / math.sqrt(k))
    st = {"kw": kw, "out": []}
    if epi == "f32":
        d = torch.empty(m, n, device="cuda")
        kw.update(epilogue=host.EPI_F32, d=d, ldd=n)
        st["out"] = [d]
    elif epi == "f16":
        n16 = n // 32 * 32
        d16, tail = torch.empty(m, n16, dtype=torch.float16, device="cuda"), torch.zeros(m, max(1, n - n16), device="cuda")
        kw.update(epilogue=host.EPI_F16, d_f16=d16, ld_f16=n16, n_f16=n16, d=tail, ldd=max(1, n - n16))
        st["out"] = [d16, tail]
    elif epi == "add_i8":
        resid = _activations(g, m, n)
        kw.update(epilogue=host.EPI_ADD_I8, resid=resid, ld_resid=n, add_scale=1.0)
        st["out"] = [resid]
    elif epi == "gelu_i8":
        d8 = torch.empty(m, n, dtype=torch.int8, device="cuda")
        kw.update(epilogue=host.EPI_GELU_I8, act_scale=1.0, d_i8=d8, ld_i8=n)
        st["out"] = [d8]
    else:
        codes = torch.zeros(host.matrix_bytes(m, n), dtype=torch.uint8, device="cuda")
        sf = torch.zeros(host.sf_bytes(m, n), dtype=torch.uint8, device="cuda")
        kw.update(epilogue=host.EPI_GELU_FP4, act_scale=1.0, d_codes=codes, d_sf=sf)
        st["out"] = [codes, sf]
        if rank > 0:                                         # the projections the next perturbed GEMM needs
            st["next_t"] = torch.zeros(m, rank, dtype=torch.int32, device="cuda")
            kw.update(next_tvec=_clt(g, pairs, rank, n), next_tvec_pair_stride=rank * n, next_nvec=rank, next_t=st["next_t"])
            st["out"].append(st["next_t"])
    return st


def _prepare_scan(case, seed):
    hidden, rows = 64 * case["heads"], case["seqs"] * case["seq"]
    g = _gen(seed)
    dt = torch.float16 if case["half"] else torch.float32
    qkv = (torch.randn(rows, 3 * hidden, device="cuda", generator=g) * 0.3).to(dt)
    beta = torch.randn(rows, device="cuda", generator=g)
    out = torch.empty(rows, hidden, dtype=dt, device="cuda")
    kw = dict(state=None, state_fp16=1, q=qkv, k=qkv[:, hidden:], v=qkv[:, 2 * hidden:], beta_raw=beta, ld_qkv=3 * hidden, ld_beta=1, beta_bias=-2.0,
              seqs_per_bias=1, hidden=hidden, heads=case["heads"], seqs=case["seqs"], T=case["seq"], method=case["method"], eps=1e-6, out=out,
              ld_out=hidden, variant=2 if case["variant"] == "per_token" else 0, qkv_f16=int(case["half"]), out_f16=int(case["half"]))
    return {"kw": kw, "out": out, "qkv": qkv}


def _prepare_update(case, seed):
    rows, cols, pairs, rank = case["rows"], case["cols"], case["pairs"], case["rank"]
    g = _gen(seed)
    w = _ternary(g, rows * cols)
    order = torch.randperm(pairs, device="cuda", generator=g).float()
    st = {"case": case, "weights": order / max(1, pairs - 1) - 0.5, "seeds": host.fill_pair_seeds(seed, 3, pairs), "w": w, "shadow": w.float(),
          "ema": torch.zeros(1, device="cuda")}
    if rank > 0:
        st["A"], st["B"] = _clt(g, pairs, rows, rank), _clt(g, pairs, rank, cols)
    return st


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("epoch", "validate"):
        return {"kind": kind, **_prepare_model(case, seed)}
    make = {"token": _prepare_token, "perturbed": _prepare_perturbed, "gemm": _prepare_gemm, "scan": _prepare_scan, "update": _prepare_update}[kind]
    return {"kind": kind, **make(case, seed)}


# ------------------------------------------------------------------------------------------------ one pass
def _run_token(st):
    c = st["case"]
    H, F, B = c["hidden"], c["hidden"] * c["mlp_mult"], c["batch"]
    s_h, s_f, sigma = 1.0 / math.sqrt(H), 1.0 / math.sqrt(F), 0.125

    def project(x, w, e, n, k, scale):
        """alpha x W^T, then the noise matrix's product added to it."""
        y = host.gemm_ternary_f_nvfp4(x[0], w[0], x[1], w[1], B, n, k, scale)
        return y if e is None else host.gemm_ternary_f_nvfp4(x[0], e[0], x[1], e[1], B, n, k, sigma * scale, 1.0, y, y)

    e = st["e"] or {"win": None, "head": None, "layers": [{"qkv": None, "ff1": None, "ff2": None}] * c["layers"]}
    w = st["w"]
    _, codes, sf = host.embedding_lookup_noise_quantize_nvfp4(st["tokens"], 1, st["emb"], st["emb_noise"], H, B, sigma, 1 if c["noisy"] else 0)
    y = project((codes, sf), w["win"], e["win"], H, H, s_h)
    x, codes, sf = host.add_pos_gelu_quantize_nvfp4(y, st["pos"], 0.8)
    _, codes, sf = host.absmean_norm_q_nvfp4(x, 1.0)
    for wl, el, S in zip(w["layers"], e["layers"], st["S"]):
        fc = 3 * H + 32
        qkv = project((codes, sf), wl["qkv"], el["qkv"], fc, H, 1.0)
        y = host.efla_step_half_qkv_fused(S, qkv, fc, -2.0, H, B, 1, 1e-6)
        _, codes, sf = host.add_scaled_to_int8_absmean_norm_q_nvfp4(x, y, 1.0, 1.0)
        if el["ff1"] is None:
            f = host.gemm_ternary_f_nvfp4_gelu_i8(codes, wl["ff1"][0], sf, wl["ff1"][1], B, F, H, s_h, 0.0, None, 1.0)
        else:
            y = host.gemm_ternary_f_nvfp4(codes, wl["ff1"][0], sf, wl["ff1"][1], B, F, H, s_h)
            f = host.gemm_ternary_f_nvfp4_gelu_i8(codes, el["ff1"][0], sf, el["ff1"][1], B, F, H, sigma * s_h, 1.0, y, 1.0)
        y = project(host.nvfp4_quantize_a(f), wl["ff2"], el["ff2"], H, F, s_f)
        _, codes, sf = host.add_scaled_to_int8_absmean_norm_q_nvfp4(x, y, 1.0, 1.0)
    logits = project((codes, sf), w["head"], e["head"], VOCAB, H, s_h)
    host.cross_entropy_loss(logits, st["bias"], None, 0.0, st["targets"], 1, st["loss"])
    return {"logits": logits, "x": x, "loss": st["loss"], "state": st["S"]}


def run(st):
    kind = st["kind"]
    if kind == "epoch":
        model = st["model"]
        model.set_tokens(st["tokens"], st["targets"])
        losses = population.es_step(model, st["seed"], st["epoch"], st["pairs"])
        st["epoch"] += 1
        out = {"losses": losses, "after": model.eval_base()}
        if st["keep"]:
            out["weights"] = model.get_weights()
        return out
    if kind == "validate":
        st["model"].set_tokens(st["tokens"], st["targets"])
        return st["model"].eval_base()
    if kind == "token":
        return _run_token(st)
    if kind == "perturbed":
        c = st["case"]
        m, k, n, rank = c["members"] * c["rows"], c["k"], c["n"], c["rank"]
        proj = dict(tvec=st["Bt"], tvec_pair_stride=rank * k, nvec=rank, t_out=st["t"]) if rank > 0 else {}
        host.rowquant(host.FE_ACT, rows=m, cols_in=k, cols_out=k, rows_per_member=c["rows"], in_f32=st["x"], ld_in=k, act_mode=0, out_codes=st["codes"],
                      out_sf=st["sf"], **proj)
        lora = dict(rank=rank, rows_per_member=c["rows"], lora_t=st["t"], t_stride=rank, lora_A=st["A"], lora_A_pair_stride=n * rank,
                    lora_scale=0.125 / math.sqrt(k) * host.c_rank(rank)) if rank > 0 else {}
        host.gemm_nvfp4_ex(a=st["codes"], b=st["b"], sfa=st["sf"], sfb=st["sfb"], m=m, n=n, k=k, alpha=1.0 / math.sqrt(k), d=st["d"], ldd=n,
                           epilogue=host.EPI_F32, **lora)
        return [st["d"], st["codes"], st["sf"]]
    if kind == "gemm":
        if "next_t" in st:
            st["next_t"].zero_()
        host.gemm_nvfp4_ex(**st["kw"])
        return st["out"]
    if kind == "scan":
        host.efla_scan(**st["kw"])
        return st["out"]
    c = st["case"]
    n = c["rows"] * c["cols"]
    if c["form"] == "dense":
        Z, sumsq = host.compute_z_sumsq(st["weights"], st["seeds"], 0x999999, n)
    else:
        Z, sumsq = host.compute_z_sumsq_lowrank(st["weights"], st["A"], st["B"], c["rows"], c["cols"], c["rank"], host.c_rank(c["rank"]))
    inv = host.update_inv_rms(sumsq, st["ema"], True, 0.95, 1e-3, n)
    host.update_shadow_ternary_device(st["w"], st["shadow"], Z, inv, 0.8, 0.008 * math.sqrt(c["pairs"]))
    return {"Z": Z, "sumsq": sumsq, "w": st["w"], "shadow": st["shadow"], "ema": st["ema"]}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _params(c):
    h, L = c["hidden"], c["layers"]
    return 2 * VOCAB * h + h * h + L * (h * h * (3 + 2 * c["mlp_mult"]) + h)


def _forward_flops(c, members):
    """Members' forward: the input projection once per distinct token of the byte vocabulary, everything else per token."""
    h, rows = c["hidden"], members * c["batch"] * c["seq"]
    per_row = c["layers"] * (2.0 * h * (h * (3 + 2 * c["mlp_mult"]) + 1) + 6.0 * h * (h // c["heads"])) + 2.0 * VOCAB * h
    return rows * per_row + 2.0 * h * h * min(rows, members * VOCAB)


def work(case):
    kind = case["kind"]
    if kind in ("epoch", "validate"):
        p, rows = _params(case), case["batch"] * case["seq"]
        if kind == "validate":
            return {"bytes": p + 4 * case["seq"] * case["hidden"] + 2 * rows + 4, "flops": _forward_flops(case, 1)}
        pairs, rank = case["pairs"], case["rank"]
        # int8 weights and fp32 shadows are read and written, the loss of every member comes out; noise is a function of the seed
        return {"bytes": 10 * p + 8 * case["seq"] * case["hidden"] + 2 * rows + 8 * pairs,
                "flops": _forward_flops(case, 2 * pairs) * (2 if rank == 0 else 1) + _forward_flops(case, 1) + 2.0 * pairs * p * max(1, rank)}
    if kind == "token":
        h, f, b, L = case["hidden"], case["hidden"] * case["mlp_mult"], case["batch"], case["layers"]
        mats = h * h + VOCAB * h + L * (3 * h * h + 2 * h * f)
        twice = 2 if case["noisy"] else 1
        return {"bytes": twice * mats * 0.5625 + L * 4.0 * b * h * h + b * (h + 4.0 * VOCAB), "flops": twice * 2.0 * b * mats + L * 6.0 * b * h * h}
    if kind == "perturbed":
        m, k, n, r = case["members"] * case["rows"], case["k"], case["n"], case["rank"]
        return {"bytes": 4.0 * m * k + 0.5625 * (m + n) * k + 4.0 * m * n, "flops": 2.0 * m * n * k + 2.0 * m * r * (n + k)}
    if kind == "gemm":
        m, n, k, r = case["m"], case["n"], case["k"], case["rank"]
        out = {"f32": 4.0, "f16": 2.0, "add_i8": 2.0, "gelu_i8": 1.0, "gelu_fp4": 0.5625}[case["epilogue"]]
        return {"bytes": 0.5625 * (m + n) * k + out * m * n + 4.0 * m * r, "flops": 2.0 * m * n * k + 2.0 * m * n * r}
    if kind == "scan":
        rows, h = case["seqs"] * case["seq"], 64 * case["heads"]
        return {"bytes": rows * ((2 if case["half"] else 4) * 4.0 * h + 4), "flops": 6.0 * rows * h * 64}
    n, pairs, rank = case["rows"] * case["cols"], case["pairs"], case["rank"]
    factors = pairs * rank * (case["rows"] + case["cols"])
    return {"bytes": 14.0 * n + factors + 12.0 * pairs, "flops": 2.0 * pairs * n * max(1, rank)}


def tolerance(case):
    kind = case["kind"]
    if kind == "epoch":
        # losses of a network of int8 / FP4 activations, and weights that follow the ranks of those losses
        return {"rel": 5e-4, "differ": 5e-3}
    if kind == "validate":
        return {"rel": 1e-4}
    if kind == "token":
        return {"rel": 2e-3, "differ": 2e-3}                 # fp16 state, int8 activations one step apart at ties
    if kind == "perturbed":
        return {"rel": 1e-5}                                 # fp32 sums of exact products; codes and scale bytes are exact
    if kind == "gemm":
        return {"f32": {"rel": 1e-5}, "f16": {"rel": 5e-4}}.get(case["epilogue"], {"differ": 1e-4})
    if kind == "scan":
        return {"rel": 2e-3}                                 # fp16 state
    return {"rel": 1e-5, "differ": 1e-5}
