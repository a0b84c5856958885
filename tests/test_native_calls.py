"""The module in front of the library's short calls (csrc/native.cpp): what it takes, what it leaves to the long way, what it refuses."""
import pytest
import torch


def test_host_tensors_and_wrong_calls_are_left_alone():
    from mpsa import _lib
    n = _lib.native()
    x = torch.zeros(1, 2, 128, 128, dtype=torch.bfloat16)
    assert n.quant_pair(x, x, 1.0, 1.0, 0, True) is None
    assert n.attention(x, x, x, None, None, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 1.0, 1.0) is None
    assert n.gemm(x, x, x, x, 1, 1, 1, 0, 0, 0, 0, 1.0, 0) is None
    for f in (n.quant_pair, n.attention, n.gemm):
        with pytest.raises(TypeError):
            f(x)


class _Sub(torch.Tensor):
    pass


def _forms(D):
    """(name, tensor [2, 3, 130, D], taken): views of every kind over one set of values."""
    g = torch.Generator(device="cuda").manual_seed(D)
    x = torch.randn(2, 3, 130, D, generator=g, device="cuda", dtype=torch.bfloat16)
    flat = torch.zeros(x.numel() + 8, device="cuda", dtype=x.dtype)
    wide = torch.zeros(2, 3, 130, D + 8, device="cuda", dtype=x.dtype)
    odd = torch.zeros(2, 3, 130, D + 4, device="cuda", dtype=x.dtype)
    dense = flat[:x.numel()].view_as(x)
    shifted = flat.clone()[1:x.numel() + 1].view_as(x)
    forms = [("dense", dense, True), ("tokens first", x.transpose(1, 2).contiguous().transpose(1, 2), True), ("padded rows", wide[..., :D], True),
             ("rows of an odd pitch", odd[..., :D], False), ("base off by one", shifted, False),
             ("depth strided", torch.zeros(2, 3, 130, 2 * D, device="cuda", dtype=x.dtype)[..., ::2], False),
             ("expanded heads", x[:, :1].expand(2, 3, 130, D), True), ("subclass", x.clone().as_subclass(_Sub), False), ("fp32", x.float(), False)]
    for name, t, taken in forms:
        if name not in ("expanded heads",):
            with torch.no_grad():
                t.copy_(x)
        yield name, t, taken


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128])
def test_every_form_gives_what_the_long_way_gives(D):
    import mpsa
    from mpsa import _lib, ops
    for name, t, taken in _forms(D):
        direct = _lib.native().quant_pair(t, t, 0.5, 1.0, 1, True)
        assert (direct is not None) == taken, name
        if name in ("rows of an odd pitch", "base off by one"):       # refused by the long way too
            with pytest.raises(ValueError):
                ops.quantize_pair(t, t, 0.5, 1.0, "e5m2")
            continue
        qc, qs, kc, ks = ops.quantize_pair(t, t, 0.5, 1.0, "e5m2")
        for codes, scales, s in ((qc, qs, 0.5), (kc, ks, 1.0)):
            ref = ops.quantize_mx(t, s, want_fp4=False, reference_format=True, kernel_format=False)
            assert torch.equal(codes.view(torch.uint8), ref.fp8) and torch.equal(scales, ref.fp8_scales), name
        out = mpsa.attention_forward(t, t, t, causal=True, out_dtype=torch.float32)
        dense = mpsa.attention_forward(t.detach().clone().contiguous(), t.contiguous(), t.contiguous(), causal=True, out_dtype=torch.float32)
        assert torch.equal(out, dense) if taken else float((out - dense).abs().max()) < 1e-2, name


@pytest.mark.gpu
def test_what_was_refused_stays_refused():
    import mpsa
    from mpsa import ops
    e = torch.zeros(1, 2, 0, 128, device="cuda", dtype=torch.bfloat16)
    x = torch.zeros(1, 2, 128, 128, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(ValueError):
        mpsa.attention_forward(e, x, x, causal=False)
    with pytest.raises(ValueError):
        ops.quantize_pair(e, x, 1.0, 1.0, "mxfp4")
    with pytest.raises(ValueError):
        mpsa.attention_forward(x.cpu(), x, x, causal=False)
    with pytest.raises(ValueError):
        mpsa.attention_forward(torch.zeros(1, 3, 128, 128, device="cuda", dtype=torch.bfloat16), x, x, causal=False)


@pytest.mark.gpu
def test_the_interpreter_is_free_during_allocation_and_launch(tmp_path):
    """A launch into a full queue, or an allocation that has to wait for the device, must not hold every other thread up: the C entries
    run without the interpreter's lock (here they are replaced by the call that tells)."""
    import ctypes
    import importlib.util
    import shutil

    from mpsa import _lib, ops
    lib, n = _lib.load(), _lib.native()
    path = tmp_path / "copy.so"                           # (its own function pointers)
    shutil.copy(n.__file__, path)
    spec = importlib.util.spec_from_file_location("copy._native", path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value
    held = address(ctypes.pythonapi.PyGILState_Check)
    m.init(address(lib.mpsa_attention_workspace), held, held, held, torch.OutOfMemoryError)
    x = torch.zeros(1, 2, 128, 128, device="cuda", dtype=torch.bfloat16)
    b = torch.zeros(128, 128, device="cuda", dtype=torch.uint8)
    status = ops.status_word(x.device).data_ptr()
    assert isinstance(m.attention(x, x, x, None, None, status, 0, 0, 1, 0, 0, 0, 1, 0, 0, 1.0, 1.0), torch.Tensor)
    assert isinstance(m.quant_pair(x, x, 1.0, 1.0, 0, True), tuple)
    assert isinstance(m.gemm(b, b, b, b, 128, 128, 128, 0, 1, 1, 0, 1.0, status), torch.Tensor)


@pytest.mark.gpu
def test_two_threads():
    import threading

    import mpsa
    from mpsa import ops
    g = torch.Generator(device="cuda").manual_seed(3)
    x = [torch.randn(1, 4, n, 128, generator=g, device="cuda", dtype=torch.bfloat16) for n in (200, 640)]

    def calls(t):
        c = mpsa.quantize_mx(t.reshape(1, 1, -1, 128), want_fp4=False)
        m, s = c.fp8.shape[2], c.fp8_sf.view(-1, 1, 32, 4, 4)
        a = c.fp8.view(m, 128)
        return [mpsa.attention_forward(t, t, t, causal=True), *ops.quantize_pair(t, t, 0.5, 1.0, "e5m2"),
                ops.gemm_block_scaled(a, s, a, s, torch.float32, m, m, 128, "mxfp8")]

    want = [calls(t) for t in x]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(40):
                    got = calls(x[i])
                    torch.cuda.current_stream().synchronize()
                    if not all(torch.equal(p.view(torch.uint8), r.view(torch.uint8)) for p, r in zip(got, want[i])):
                        wrong.append((i, "other results"))
        except Exception as e:                            # noqa: BLE001 (reported by the test)
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:4]


@pytest.mark.gpu
@pytest.mark.parametrize("flag", ["numpy", "float", "int"])
def test_truth_values_of_any_kind(flag):
    import numpy as np
    import mpsa
    x = torch.randn(1, 2, 130, 128, device="cuda", dtype=torch.bfloat16)
    for value in (False, True):
        given = {"numpy": np.bool_, "float": float, "int": int}[flag](value)
        got = mpsa.attention_forward(x, x, x, causal=given, smooth_k=given)
        assert torch.equal(got, mpsa.attention_forward(x, x, x, causal=value, smooth_k=value))


@pytest.fixture
def no_module(monkeypatch, tmp_path):
    """As on a machine without a C++ compiler and without a built module."""
    from mpsa import _lib
    monkeypatch.setattr(_lib, "_native", None)
    real = _lib._module

    def module(name, path):
        mod = real(name, path)
        if name == "_mpsa_build":
            mod.native_out = lambda: str(tmp_path / "absent.so")
        return mod
    monkeypatch.setattr(_lib, "_module", module)
    monkeypatch.setenv("CXX", str(tmp_path / "no-compiler"))
    with pytest.warns(RuntimeWarning, match="not available"):
        n = _lib.native()
    assert _lib.native() is n                             # (asked for once)
    return n


def test_without_the_module_every_call_is_left_to_the_long_way(no_module):
    assert [no_module.attention(1), no_module.quant_pair(2, 3), no_module.gemm()] == [None] * 3


def test_build_without_the_module_still_builds_the_library(tmp_path):
    import os
    import shutil
    import subprocess
    import sys

    from mpsa import _lib
    here = os.path.dirname(os.path.dirname(_lib.lib_path()))
    top = tmp_path / "package"
    (top / "mpsa").mkdir(parents=True)
    shutil.copytree(os.path.join(here, "csrc"), top / "csrc")
    shutil.copytree(os.path.join(os.path.dirname(here), "include"), tmp_path / "include")
    shutil.copy(os.path.join(here, "build.py"), top / "build.py")
    lib = top / "mpsa" / "libmpsa.so"                     # up to date: nothing to compile
    lib.write_bytes(b"")
    r = subprocess.run([sys.executable, str(top / "build.py")], env=dict(os.environ, CXX=str(tmp_path / "no-compiler")), capture_output=True, text=True)
    assert r.returncode == 0 and str(lib) in r.stdout and "not built" in r.stderr, (r.stdout, r.stderr)


def test_the_module_is_that_of_this_python_and_torch():
    import sysconfig

    from mpsa import _lib
    name = _lib.native().__file__
    assert torch.__version__ in name and sysconfig.get_config_var("SOABI") in name


@pytest.mark.gpu
def test_calls_without_the_module(no_module, monkeypatch):
    import mpsa
    from mpsa import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.randn(1, 4, 300, 128, generator=g, device="cuda", dtype=torch.bfloat16)
    c = mpsa.quantize_mx(x[:, :, :256].reshape(1, 1, -1, 128), want_fp4=False)
    m, s = c.fp8.shape[2], c.fp8_sf.view(-1, 1, 32, 4, 4)
    a = c.fp8.view(m, 128)

    def calls():
        kv = mpsa.prepare_kv(x, x, pv_mode="requant")
        return [*ops.quantize_pair(x, x, 0.5, 1.0, "mxfp4"), *ops.quantize_pair(x, x, 0.5, 1.0, "e5m2"),
                ops.gemm_block_scaled(a, s, a, s, torch.float32, m, m, 128, "mxfp8"),
                mpsa.attention_forward(x, x, x, causal=True), mpsa.attention_forward(x, x, x, causal=False, pv_mode="requant", smooth_k=True),
                mpsa.attention_forward(x, x, x, causal=True, pv_mode="requant", router="online", tau=1.1),
                mpsa.attention_forward(x, x, x, causal=False, fp4_kind="nvfp4"), mpsa.attention_forward(x, None, None, causal=True, kv=kv)]

    got = calls()
    monkeypatch.undo()
    assert _lib.native().__file__
    for i, (p, r) in enumerate(zip(got, calls())):
        assert torch.equal(p.view(torch.uint8), r.view(torch.uint8)), i
