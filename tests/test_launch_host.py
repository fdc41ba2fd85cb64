"""The host's side of a launch (native/csrc/launch.cpp): what its checks accept and refuse, and products on two streams and threads."""
import ctypes
import os
import subprocess
import sys
import threading

import pytest
import torch

from atom_b200 import native


def test_checks_of_type_sizes_and_strides():
    native._host()
    x = torch.zeros(4, 6, 8, dtype=torch.bfloat16)
    cut, turned = x[:, :, :4], x.transpose(1, 2)
    assert native._dense(x, native.BF16) and native._dense(x, None, 4, 6, 8) and native._dense(x, cut, None, 6, None)
    assert not native._dense(x, native.F32) and not native._dense(x, native.BF16, 4, 6) and not native._dense(x, None, 4, 7, 8)
    assert not native._dense(x, torch.zeros(1)) and not native._dense(cut, None) and not native._dense(turned, None)
    assert native._rows(cut, native.BF16, 4, 6, 4) and not native._rows(turned, None) and not native._rows(cut, native.I32)
    assert native._dense(torch.zeros(3, dtype=torch.int32), native.I32, 3) and not native._dense(torch.zeros(3, dtype=torch.int64), native.I32)
    assert native._rows16(x[0]) and not native._rows16(x[0][:, 1:]) and not native._rows16(torch.zeros(2, 5, dtype=torch.bfloat16))


def test_refusals():
    native._host()
    x = torch.zeros(4, 64, dtype=torch.bfloat16)
    native._cuda(None, None)
    with pytest.raises(native.NativeError):
        native._cuda(None, x)
    with pytest.raises(native.NativeError):
        native.gemm_bf16(x, x, x)
    with pytest.raises(native.NativeError):
        native.gemm_batched(x, x, x)
    with pytest.raises(TypeError):
        native._cuda(3)
    fn = native.lib().atom_gemm_rows_supports
    assert fn(16, 64, 64, 64) in (0, 1)
    for args in ((16, 64, 64), (16, 64, 64, 64, 1), (16, 64, 64, None), (16, 64, 64, 2.5)):
        with pytest.raises(TypeError):
            fn(*args)
    with pytest.raises(TypeError):      # a tensor that must be there: nothing is launched
        native.lib().atom_relu2(None, 1, 0, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_products_on_two_streams_and_threads(out_dtype):
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    a, w = r(70, 256), r(192, 256)
    ab, wb = r(70, 4, 64), r(4, 96, 64)
    want, want_b = (a.double() @ w.double().T), torch.einsum("mbk,bnk->mbn", ab.double(), wb.double())
    tol = 2.0 ** -8 if out_dtype == torch.bfloat16 else 64 * 2.0 ** -23      # (half a unit of bf16; sums of 256 in 32-bit)
    torch.cuda.synchronize()

    def work(stream, got):
        with torch.cuda.stream(stream):
            for _ in range(50):
                out, out_b = torch.empty(70, 192, dtype=out_dtype, device="cuda"), torch.empty(70, 4, 96, dtype=out_dtype, device="cuda")
                native.gemm_bf16(out, a, w)
                native.gemm_batched(out_b, ab, wb)
                got.append((out, out_b))
        stream.synchronize()

    results = [[], []]
    threads = [threading.Thread(target=work, args=(torch.cuda.Stream(), x)) for x in results]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for got in results:
        assert len(got) == 50
        for out, out_b in got:
            assert (out.double() - want).abs().max() <= tol * want.abs().max()
            assert (out_b.double() - want_b).abs().max() <= tol * want_b.abs().max()
    for bad in ((a[:, 1:], w), (a, w[:, :255]), (a.float(), w), (a, w.T)):
        with pytest.raises(AssertionError):
            native.gemm_bf16(torch.empty(70, 192, dtype=out_dtype, device="cuda"), *bad)
    with pytest.raises(AssertionError):
        native.gemm_bf16(torch.empty(192, 70, dtype=out_dtype, device="cuda").T, a, w)
    with pytest.raises(native.NativeError):
        native.gemm_bf16(torch.empty(70, 192, dtype=torch.float16, device="cuda"), a, w)


def test_a_tensor_without_memory_is_an_error_of_python():
    with pytest.raises(RuntimeError):
        native.lib().atom_relu2(torch.zeros(2, 2).to_sparse(), 1, 0, 0)


class _OnDevice(torch.Tensor):
    """Host memory that says that it lies on a device."""
    is_cuda = True


def test_memory_that_is_not_pinned_is_not_read_by_a_kernel(monkeypatch):
    launched = []

    class Lib:
        atom_step_arrays_tables = staticmethod(lambda: 8)
        atom_step_arrays = staticmethod(lambda *args: launched.append(args) or 0)

    monkeypatch.setattr(native, "lib", Lib)
    monkeypatch.setattr(native, "_stream", lambda: 0)
    src, dst = torch.zeros(16, dtype=torch.int32), torch.zeros(64, dtype=torch.int32).as_subclass(_OnDevice)
    with pytest.raises(native.NativeError):
        native.step_arrays(dst, src, 4, 2, [3], [8], [5])
    assert not launched


def test_a_kernel_writes_into_no_other_tensors_memory():
    """A copy that is made when it is first written to is made before a function has its address."""
    got = []
    relu2 = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int64, ctypes.c_void_p)
    fn = relu2(lambda x, dtype, n, stream: got.append(x) or 0)
    bound = native._host().bind(ctypes.cast(fn, ctypes.c_void_p).value, "IPILP", "relu2")
    x = torch.ones(4)
    late = torch._lazy_clone(x)
    assert bound(late, native.F32, 4, 0) == 0
    assert got == [late.data_ptr()] and got != [x.data_ptr()]


def test_one_module_whatever_is_imported_first():
    """What the module is built from does not change when the sampler comes, and a library that was loaded before it calls the
    sampler's functions through the module too."""
    code = """
import ctypes
from atom_b200 import native
before, lib = native.signatures(), native.lib()
from atom_b200.sampling import sampler
assert native.signatures() == before, set(native.signatures()) ^ set(before)
plain = [n for n in native._SIGNATURES if isinstance(getattr(lib, n), ctypes._CFuncPtr)]
assert not plain, plain
assert callable(lib.atom_sample) and type(lib.atom_sample) is type(lib.atom_relu2)
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=900)
    assert p.returncode == 0, p.stderr[-2000:]


def test_the_library_is_given_out_when_its_functions_are_bound(monkeypatch):
    """Another thread that asks for the library while it is being bound (the module may be compiled then) does not get half of it."""
    native.lib()
    declare, seen = native._declare, []
    monkeypatch.setattr(native, "_lib", None)
    monkeypatch.setattr(native, "_declare", lambda l: (seen.append(native._lib), declare(l)))
    assert type(native.lib().atom_relu2) is type(native.lib().atom_gemm_bf16) and seen == [None]
