"""Host-side mirror of the reference's kernel-entry interface (namespaces bitnet_cuda / efla_lm_cuda of
the reference's src/cuda_kernels.h and src/efla_lm_kernels.h), on torch device tensors.

Function names and argument meaning follow the reference; every call goes through the C ABI of
libbnf4.so on the current CUDA stream. torch is used for device memory and streams only.

The functions that a token loop calls dozens of times per token go through the extension _host, which converts arguments, allocates the
outputs and calls the library natively (8.5 us per call through ctypes, more than the kernels take).
"""
from __future__ import annotations

import ctypes as C

import torch

from . import lib as _l

FE_INT8, FE_WQKV, FE_EMBED_DENSE, FE_EMBED_LOWRANK, FE_POS_GELU, FE_POS_GELU_ABSMEAN, FE_ACT, FE_ABSMEAN, FE_ADD_ABSMEAN = range(9)
EPI_F32, EPI_GELU_I8, EPI_GELU_FP4, EPI_ADD_I8, EPI_F16 = range(5)

C_RANK_BASE = 0.6123724356957945  # sqrt(3/8)


def c_rank(rank: int) -> float:
    """Normalisation of a rank-r perturbation: sqrt(3/8)/sqrt(r), evaluated in fp32 like the library does."""
    import numpy as np
    return 0.0 if rank <= 0 else float(np.float32(C_RANK_BASE) / np.sqrt(np.float32(rank)))


_stream = _l.stream
_native = None


def _n():
    """The native call path. Raises if it has not been built, like lib.load()."""
    global _native
    if _native is None:
        _l.load()
        try:
            from . import _host
        except ImportError as e:
            raise _l.Bnf4Error(f"the extension _host cannot be loaded ({e}): build it with `python -m bitnet_nvfp4_b200.build`") from e
        _host.set_error_class(_l.Bnf4Error)
        codes = {C.c_void_p: "P", C.c_int: "i", C.c_float: "f", C.c_longlong: "q"}
        for kind, desc in enumerate((_l.RowQuantDesc, _l.GemmDesc, _l.EflaDesc)):
            _host.register_desc(kind, C.sizeof(desc), [(name, getattr(desc, name).offset, codes[t]) for name, t in desc._fields_])
        _native = _host
    return _native


def _p(t):
    return None if t is None else t.data_ptr()


def sf_bytes(rows: int, k: int) -> int:
    """bnf4_nvfp4_sfa_bytes: whole atoms of 128 rows x 64 elements, one byte per 16 elements."""
    return -(-rows // 128) * 128 * (-(-(-(-k // 16)) // 4) * 4)


def matrix_bytes(rows: int, cols: int) -> int:
    """bnf4_nvfp4_matrix_bytes: two elements per byte."""
    return (rows * cols * 4 + 7) // 8


def _alloc_q(like: torch.Tensor, rows: int, cols: int, want_q=True):
    """Outputs of a quantiser on the device of `like`. Nothing is cleared: the library writes every int8 value, code and scale byte, the
    padding of the scale array included."""
    q = torch.empty((rows, cols), dtype=torch.int8, device=like.device) if want_q else None
    return q, *(torch.empty(n, dtype=torch.uint8, device=like.device) for n in (matrix_bytes(rows, cols), sf_bytes(rows, cols)))


def device_error() -> int:
    code = C.c_int(0)
    _l.check(_l.load().bnf4_device_error(_stream(), C.byref(code)))
    return code.value


# ------------------------------------------------------------------------------------------ quantisers
# (of a quantiser's outputs, codes and scale bytes -- one operand of a GEMM -- may share a storage: keeping either keeps both)
def nvfp4_quantize_a(x: torch.Tensor, k_out: int | None = None):
    return _n().quantize_a(x, k_out or x.shape[1])


def nvfp4_quantize_b(w: torch.Tensor, k_out: int | None = None):
    n, k_in = w.shape
    k_out = k_out or k_in
    _, codes, sf = _alloc_q(w, n, k_out, want_q=False)
    _l.check(_l.load().bnf4_nvfp4_quantize_b(_p(w), 1, n, k_in, k_out, _p(codes), _p(sf), _stream()))
    return codes, sf


def nvfp4_quantize_f32(x: torch.Tensor, k_out: int | None = None):
    """fp32 rows straight to NVFP4 (no int8 stage)."""
    m, k_in = x.shape
    k_out = k_out or k_in
    _, codes, sf = _alloc_q(x, m, k_out, want_q=False)
    if m % 128 or k_out % 64:
        sf.zero_()  # (this kernel leaves the padding alone)
    _l.check(_l.load().bnf4_nvfp4_quantize_f32(_p(x), m, k_in, k_out, _p(codes), _p(sf), _stream()))
    return codes, sf


def nvfp4_quantize_wqkv_fused(wq, wk, wv, wb, hidden: int, rows_total: int, scale: float):
    codes = torch.zeros(matrix_bytes(rows_total, hidden), dtype=torch.uint8, device=wq.device)
    sf = torch.zeros(sf_bytes(rows_total, hidden), dtype=torch.uint8, device=wq.device)
    _l.check(_l.load().bnf4_nvfp4_quantize_wqkv_fused(_p(wq), _p(wk), _p(wv), _p(wb), 1, hidden, hidden, rows_total, scale,
                                                      scale, scale, scale, _p(codes), _p(sf), _stream()))
    return codes, sf


def embedding_lookup_noise_quantize_nvfp4(tokens_t, token_stride, emb_w, emb_noise, hidden, batch, noise_scale, anti_sign):
    return _n().embedding_lookup_noise_quantize(tokens_t, token_stride, emb_w, emb_noise, hidden, batch, noise_scale, anti_sign)


def add_pos_gelu_quantize_nvfp4(x, pos_t, act_scale):
    return _n().add_pos_gelu_quantize(x, pos_t, act_scale)


def activation_quantize_nvfp4(x, cols_out, activation):
    rows, cols_in = x.shape
    q, codes, sf = _alloc_q(x, rows, cols_out)
    _l.check(_l.load().bnf4_activation_quantize_nvfp4(_p(x), rows, cols_in, cols_out, activation, _p(q), _p(codes), _p(sf),
                                                      _stream()))
    return q, codes, sf


def gelu_quantize_nvfp4(x, cols_out, act_scale):
    rows, cols_in = x.shape
    q, codes, sf = _alloc_q(x, rows, cols_out)
    _l.check(_l.load().bnf4_gelu_quantize_nvfp4(_p(x), rows, cols_in, cols_out, act_scale, _p(q), _p(codes), _p(sf), _stream()))
    return q, codes, sf


def absmean_norm_q_nvfp4(x8, scale):
    return _n().absmean_norm_q(x8, scale)


def add_scaled_to_int8_absmean_norm_q_nvfp4(x8_inout, y, add_scale, norm_scale):
    return _n().add_scaled_absmean_norm_q(x8_inout, y, add_scale, norm_scale)


def rowquant(front_end: int, **kw):
    """Generic row quantiser (bnf4_rowquant); keyword names are the fields of bnf4_rowquant_desc,
    tensors are converted to device pointers."""
    _n().desc_call(0, front_end, kw)


# ------------------------------------------------------------------------------------------ GEMM
def gemm_ternary_f_nvfp4(a, b, sfa, sfb, m, n, k, alpha, beta=0.0, c=None, d=None):
    return _n().gemm(a, b, sfa, sfb, m, n, k, alpha, beta, c, d)


def gemm_ternary_f_nvfp4_gelu_i8(a, b, sfa, sfb, m, n, k, alpha, beta, c, act_scale):
    return _n().gemm_gelu_i8(a, b, sfa, sfb, m, n, k, alpha, beta, c, act_scale)


def gemm_nvfp4_ex(**kw):
    """Full-form GEMM (bnf4_gemm_nvfp4_ex); keyword names are the fields of bnf4_gemm_desc."""
    _n().desc_call(1, 0, kw)


# ------------------------------------------------------------------------------------------ ternary GEMM / rank-r helpers
def gemm_ternary_f(x, w, scale_x, out_scale):
    batch, cols = x.shape
    rows = w.shape[0]
    out = torch.empty((batch, rows), dtype=torch.float32, device=x.device)
    _l.check(_l.load().bnf4_gemm_ternary_f(_p(x), _p(w), _p(scale_x), rows, cols, batch, out_scale, _p(out), _stream()))
    return out


def lora_compute_t(x, B, rank):
    batch, cols = x.shape
    t = torch.empty((batch, rank), dtype=torch.int32, device=x.device)
    _l.check(_l.load().bnf4_lora_compute_t(_p(x), _p(B), cols, batch, rank, _p(t), _stream()))
    return t


def lora_add(t, A, rows, scale, out):
    batch, rank = t.shape
    _l.check(_l.load().bnf4_lora_add(_p(t), _p(A), rows, batch, rank, scale, _p(out), _stream()))
    return out


def split_qkvb_fused(qkv, hidden, beta_bias):
    batch, fused_cols = qkv.shape
    q, k, v = (torch.empty((batch, hidden), dtype=torch.float32, device=qkv.device) for _ in range(3))
    beta = torch.empty(batch, dtype=torch.float32, device=qkv.device)
    _l.check(_l.load().bnf4_split_qkvb_fused(_p(qkv), batch, hidden, fused_cols, _p(q), _p(k), _p(v), _p(beta), beta_bias,
                                             _stream()))
    return q, k, v, beta


# ------------------------------------------------------------------------------------------ EFLA
def efla_scan(**kw):
    """Whole-sequence scan / generic recurrence (bnf4_efla_scan); keyword names are the fields of bnf4_efla_desc."""
    _n().desc_call(2, 0, kw)


def efla_step_half_qkv_fused(S, qkv, fused_cols, beta_bias, hidden, batch, method, eps):
    return _n().efla_step_half(S, qkv, fused_cols, beta_bias, hidden, batch, method, eps)


def efla_step_qkv_fused(S, qkv, fused_cols, beta_bias, hidden, batch, method, eps):
    if qkv.is_floating_point() and qkv.dtype != torch.float32:
        raise TypeError(f"qkv must be float32, not {qkv.dtype}")
    out = qkv.new_empty((batch, hidden), dtype=torch.float32)
    _l.check(_l.load().bnf4_efla_step_qkv_fused(_p(S), _p(qkv), fused_cols, beta_bias, hidden, batch, method, eps, _p(out),
                                                _stream()))
    return out


# ------------------------------------------------------------------------------------------ loss / noise / update
def cross_entropy_loss(logits, bias, bias_noise, bias_noise_scale, targets_t, token_stride, loss_accum):
    _n().cross_entropy(logits, bias, bias_noise, bias_noise_scale, targets_t, token_stride, loss_accum)


def cross_entropy_population(logits, ld, bias, bias_noise_i8, sigma, targets, vocab, members, rows_per_member):
    partial = torch.empty(members * 16, dtype=torch.float32, device=logits.device)
    loss = torch.empty(members, dtype=torch.float32, device=logits.device)
    _l.check(_l.load().bnf4_cross_entropy_population(_p(logits), ld, _p(bias), _p(bias_noise_i8), sigma, _p(targets), vocab,
                                                     members, rows_per_member, _p(partial), _p(loss), _stream()))
    return loss


def fill_ternary_noise(n, seed, use_clt=True, clt_k=4, device="cuda"):
    out = torch.empty(n, dtype=torch.int8, device=device)
    _l.check(_l.load().bnf4_fill_ternary_noise(_p(out), n, seed, int(use_clt), clt_k, _stream()))
    return out


def fill_pair_seeds(base_seed, epoch, pairs, device="cuda"):
    out = torch.empty(pairs, dtype=torch.int64, device=device)
    _l.check(_l.load().bnf4_fill_pair_seeds(base_seed, epoch, pairs, _p(out), _stream()))
    return out


def compute_z_sumsq(pair_weights, pair_seeds, salt, n, use_clt=True, clt_k=4):
    Z = torch.empty(n, dtype=torch.float32, device=pair_weights.device)
    sumsq = torch.zeros(1, dtype=torch.float32, device=pair_weights.device)
    _l.check(_l.load().bnf4_compute_z_sumsq(_p(pair_weights), _p(pair_seeds), salt, pair_weights.numel(), n, int(use_clt),
                                            clt_k, _p(Z), _p(sumsq), _stream()))
    return Z, sumsq


def compute_z_sumsq_lowrank(pair_weights, A, B, rows, cols, rank, cscale):
    pairs = pair_weights.numel()
    Z = torch.empty(rows * cols, dtype=torch.float32, device=pair_weights.device)
    sumsq = torch.zeros(1, dtype=torch.float32, device=pair_weights.device)
    _l.check(_l.load().bnf4_compute_z_sumsq_lowrank(_p(pair_weights), _p(A), rows * rank, _p(B), rank * cols, pairs, rows, cols,
                                                    rank, cscale, _p(Z), _p(sumsq), _stream()))
    return Z, sumsq


def update_inv_rms(sumsq, rms_ema, use_adaptive, beta, eps, n):
    inv = torch.empty(1, dtype=torch.float32, device=sumsq.device)
    _l.check(_l.load().bnf4_update_inv_rms(_p(sumsq), _p(rms_ema), int(use_adaptive), beta, eps, n, _p(inv), _stream()))
    return inv


def update_shadow_ternary_device(w, shadow, Z, inv_rms, lr, thresh):
    _l.check(_l.load().bnf4_update_shadow_ternary_device(_p(w), _p(shadow), _p(Z), Z.numel(), _p(inv_rms), lr, thresh, _stream()))


FITNESS_SIGN, FITNESS_ZSCORE, FITNESS_CENTERED_RANK = 0, 1, 2  # the reference's TrainConfig::FitnessMode values


def shape_pair_weights(w_host, mode=FITNESS_CENTERED_RANK, clip=3.0):
    """Host-side fitness shaping on a float32 numpy array (in place); mode as in the reference's FitnessMode enum."""
    import numpy as np
    assert w_host.dtype == np.float32 and w_host.flags["C_CONTIGUOUS"]
    _l.check(_l.load().bnf4_shape_pair_weights(w_host.ctypes.data, w_host.size, mode, clip))
    return w_host
