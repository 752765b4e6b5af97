"""The native per-call path behind host.py: conversions, outputs, errors and threads, against direct calls of the C ABI."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import torch
    from bitnet_nvfp4_b200 import host
    assert torch.cuda.is_available()
    return host


def test_outputs_match_the_c_abi(H):
    import torch
    from bitnet_nvfp4_b200 import lib
    x = torch.from_numpy(np.random.default_rng(1).integers(-127, 128, (33, 80)).astype(np.int8)).cuda()
    codes, sf = H.nvfp4_quantize_a(x, 96)
    c2, s2 = torch.empty_like(codes), torch.empty_like(sf)
    assert codes.numel() == H.matrix_bytes(33, 96) and sf.numel() == H.sf_bytes(33, 96) and codes.device == x.device
    lib.check(lib.load().bnf4_nvfp4_quantize_a(x.data_ptr(), 33, 1, 80, 96, c2.data_ptr(), s2.data_ptr(), lib.stream()))
    assert torch.equal(codes, c2) and torch.equal(sf, s2)
    d = torch.zeros((33, 33), device="cuda")
    assert H.gemm_ternary_f_nvfp4(codes[: H.matrix_bytes(33, 64)], codes[: H.matrix_bytes(33, 64)], sf, sf, np.int64(33), 33, 64, 1, d=d) is d
    assert H.gemm_ternary_f_nvfp4(codes, codes, sf, sf, 33, 33, 64, 1.0).shape == (33, 33)


def test_descriptor_fields_of_every_type(H):
    """Pointers as tensors, integers and None, 32- and 64-bit integers, floats from ints; names that are no fields are ignored."""
    import torch
    from bitnet_nvfp4_b200 import lib
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randint(-127, 128, (8, 64), dtype=torch.int8, device="cuda", generator=g)
    tv = torch.randint(-4, 5, (2, 1, 64), dtype=torch.int8, device="cuda", generator=g)
    got = []
    for native in (True, False):
        codes, sf, t = torch.zeros(256, dtype=torch.uint8, device="cuda"), torch.zeros(512, dtype=torch.uint8, device="cuda"), torch.zeros(8, dtype=torch.int32, device="cuda")
        kw = dict(rows=np.int32(8), cols_in=64, cols_out=64, rows_per_member=2, in_i8=x.data_ptr(), ld_in=64, norm_scale=3, out_q=None, out_codes=codes, out_sf=sf,
                  tvec=tv, tvec_pair_stride=64, nvec=True, t_out=t)
        if native:
            H.rowquant(H.FE_ABSMEAN, no_such_field=1, **kw)
        else:
            d = lib.RowQuantDesc()
            for k, v in kw.items():
                setattr(d, k, v.data_ptr() if isinstance(v, torch.Tensor) else int(v) if isinstance(v, np.integer) else v)
            lib.check(lib.load().bnf4_rowquant(H.FE_ABSMEAN, C.byref(d), lib.stream()))
        got.append((codes, sf, t))
    assert all(torch.equal(a, b) for a, b in zip(*got))


def test_errors(H):
    import torch
    from bitnet_nvfp4_b200.lib import Bnf4Error
    x = torch.zeros((4, 64), dtype=torch.int8, device="cuda")
    with pytest.raises(Bnf4Error):
        H.nvfp4_quantize_a(x, 72)            # no multiple of 16
    with pytest.raises(ValueError):
        H.absmean_norm_q_nvfp4(x.view(-1), 1.0)
    with pytest.raises(TypeError):
        H.absmean_norm_q_nvfp4(x, "1.0")
    with pytest.raises(TypeError):
        H.rowquant(H.FE_ABSMEAN, rows=1.5)
    with pytest.raises(Bnf4Error):
        H.gemm_nvfp4_ex(m=1, n=1, k=63)


def test_threads_use_their_own_streams(H):
    import torch
    x = [torch.full((64, 512), i + 1, dtype=torch.int8, device="cuda") for i in range(4)]
    ref = [H.absmean_norm_q_nvfp4(t, 8.0) for t in x]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(200):
                out = H.absmean_norm_q_nvfp4(x[i], 8.0)
            torch.cuda.current_stream().synchronize()
            if not all(torch.equal(a[: 64 * 32], b[: 64 * 32]) for a, b in zip(out, ref[i])):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad


@pytest.mark.parametrize("state_half", [True, False])
def test_single_step_output_is_fp32_whatever_holds_the_inputs(H, state_half):
    """The kernel writes 4 * batch * hidden bytes. Halves, which it would read as floats, are refused; raw bytes of floats are taken."""
    import torch
    step = H.efla_step_half_qkv_fused if state_half else H.efla_step_qkv_fused
    qkv = torch.randn(4, 3 * 64 + 32, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    def state():
        return torch.zeros(4, 64, 64, dtype=torch.float16 if state_half else torch.float32, device="cuda")
    want = step(state(), qkv, 224, -2.0, 64, 4, 1, 1e-6)
    for raw in (qkv.view(torch.uint8), qkv.view(torch.int32)):
        got = step(state(), raw, 224, -2.0, 64, 4, 1, 1e-6)
        assert got.dtype == torch.float32 and torch.equal(got, want)
    for dt in (torch.float16, torch.bfloat16, torch.float64):
        with pytest.raises(TypeError):
            step(state(), qkv.to(dt), 224, -2.0, 64, 4, 1, 1e-6)


class Raw:
    """Device memory as another library hands it out: an address, a shape and a device."""

    def __init__(self, t):
        self.t, self.shape, self.device = t, tuple(t.shape), t.device

    def data_ptr(self):
        return self.t.data_ptr()


def test_objects_that_are_no_tensors(H):
    """Arguments are taken by their data_ptr(), descriptor fields also as ctypes values, as the ctypes structures take them."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randint(-127, 128, (32, 128), dtype=torch.int8, device="cuda", generator=g)
    y = torch.randn(32, 128, device="cuda", generator=g)
    for f, args in ((H.nvfp4_quantize_a, (x,)), (H.nvfp4_quantize_b, (x,)), (H.absmean_norm_q_nvfp4, (x, 1.0)), (H.add_pos_gelu_quantize_nvfp4, (y, y, 0.8)),
                    (H.gelu_quantize_nvfp4, (y, 128, 0.8)), (H.activation_quantize_nvfp4, (y, 128, 1))):
        want = f(*args)
        got = f(*(Raw(a) if isinstance(a, torch.Tensor) else a for a in args))
        assert all(b is None or (torch.equal(a, b) and a.device == x.device) for a, b in zip(got, want))
    codes, sf = H.nvfp4_quantize_a(x)
    d = torch.zeros(32, 32, device="cuda")
    out = Raw(d)
    assert H.gemm_ternary_f_nvfp4(Raw(codes), Raw(codes), Raw(sf), Raw(sf), 32, 32, 128, 1.0, d=out) is out
    assert torch.equal(d, H.gemm_ternary_f_nvfp4(codes, codes, sf, sf, 32, 32, 128, 1.0)) and d.any()
    c2, s2 = torch.zeros_like(codes), torch.zeros_like(sf)
    H.rowquant(H.FE_INT8, rows=C.c_int(32), cols_in=128, cols_out=128, in_i8=C.c_void_p(x.data_ptr()), ld_in=128, out_codes=Raw(c2), out_sf=s2, out_q=C.c_void_p(),
               norm_scale=C.c_float(1.0), tvec_pair_stride=C.c_longlong(0))
    assert torch.equal(c2, codes) and torch.equal(s2, sf)
    for bad in (dict(rows=1.5), dict(rows="8"), dict(in_i8=1.5), dict(in_i8=b"x"), dict(norm_scale="1")):
        with pytest.raises(TypeError):
            H.rowquant(H.FE_INT8, **{**dict(rows=32, cols_in=128, cols_out=128, in_i8=x, ld_in=128, out_codes=c2, out_sf=s2), **bad})


def test_quantised_values_have_their_own_storage(H):
    """They can be kept, saved or grown without the operand, whose codes and scale bytes share one."""
    import io

    import torch
    x = torch.randint(-127, 128, (33, 128), dtype=torch.int8, device="cuda")
    q, codes, sf = H.absmean_norm_q_nvfp4(x, 1.0)
    assert q.untyped_storage().nbytes() == q.numel() == 33 * 128 and q.storage_offset() == 0 and q.is_contiguous()
    assert codes.untyped_storage().data_ptr() == sf.untyped_storage().data_ptr() != q.untyped_storage().data_ptr()
    assert codes.untyped_storage().nbytes() < codes.numel() + sf.numel() + 512 and sf.data_ptr() >= codes.data_ptr() + codes.numel() and sf.data_ptr() % 512 == 0
    want, other = q.clone(), codes.clone()
    buf = io.BytesIO()
    torch.save(q, buf)
    assert buf.tell() < q.numel() + 2048 and torch.equal(torch.load(io.BytesIO(buf.getvalue())), q)
    q.resize_(100, 128)
    q[33:].fill_(5)
    assert torch.equal(q[:33], want) and torch.equal(codes, other)
    q.record_stream(torch.cuda.Stream())
    sf.record_stream(torch.cuda.Stream())
    with torch.inference_mode():
        assert H.nvfp4_quantize_a(x)[0].is_inference()
    assert H.nvfp4_quantize_a(x[:0])[0].numel() == 0
