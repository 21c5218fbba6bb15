"""The call layer of the op-level entry points (host/fastcall.c) and its stand-in through ctypes: the same return codes, error texts and
treatment of arguments, without a GPU (every call is refused before it reaches one)."""
import ctypes as C
import importlib.machinery
import sys
import types

import numpy as np
import pytest

from bonsai_vk_b200 import BonsaiError, Buffer, Context, build, lib

CALLS = {"bn_act_quant_q81": 6, "bn_gemv_q81": 11, "bn_gemm_act_quant": 11, "bn_gemm_q81": 12, "bn_attn_insert": 18, "bn_attn_attend": 11}


@pytest.fixture(params=["native", "ctypes"])
def layer(request, monkeypatch):
    build.build_lib()
    build.build_fastcall()
    L = lib.load_library()
    if request.param == "ctypes":
        monkeypatch.setitem(sys.modules, "bonsai_vk_b200._fastcall", None)
        monkeypatch.delattr(sys.modules["bonsai_vk_b200"], "_fastcall", raising=False)
    return L, lib._call_layer(L, L._bn_signatures)


@pytest.mark.parametrize("name", CALLS)
def test_null_context_is_refused(layer, name):
    L, fast = layer
    assert getattr(fast, name)(*([0] * CALLS[name])) == -2
    assert L.bn_last_error().decode() == f"{name}: null context"


@pytest.mark.parametrize("name", CALLS)
def test_arguments_are_checked(layer, name):
    _, fast = layer
    with pytest.raises((TypeError, C.ArgumentError)):
        getattr(fast, name)(*([0] * (CALLS[name] - 1)))
    with pytest.raises(C.ArgumentError):
        getattr(fast, name)(*([0] * (CALLS[name] - 1) + [0.5]))


@pytest.mark.parametrize("number", [5, True, np.int64(5), np.array(5), 2 ** 70, -1])
def test_whole_numbers_are_taken(layer, number):
    _, fast = layer
    assert fast.bn_act_quant_q81(0, 0, number, number, 0, number) == -2


def test_ctypes_numbers_are_taken(layer):
    """An instance of the parameter's own ctypes type is one of its values; of another type it is refused."""
    _, fast = layer
    assert fast.bn_act_quant_q81(C.c_void_p(), 0, C.c_size_t(64), C.c_int(512), C.c_void_p(), 0) == -2
    with pytest.raises(C.ArgumentError):
        fast.bn_act_quant_q81(0, 0, C.c_int(64), 512, 0, 0)


class _Short(C.Structure):
    _fields_ = [("n_head", C.c_int32)]


class _Longer(lib.AttnDimsC):
    _fields_ = [("more", C.c_int32)]


@pytest.mark.parametrize("dims,refusal", [
    (lib.AttnDimsC(), None), (_Longer(), None),
    (lib.HParamsC(), C.ArgumentError), (_Short(), C.ArgumentError), (C.c_int(16), C.ArgumentError), (C.pointer(lib.AttnDimsC()), C.ArgumentError),
    ((lib.AttnDimsC * 2)(), C.ArgumentError), (None, TypeError), (16, TypeError)])
def test_attention_takes_its_own_dims_only(layer, dims, refusal):
    """Only an AttnDimsC may be read as sizes; a call that gets that far is refused for its null context."""
    L, fast = layer
    c, b = types.SimpleNamespace(fast=fast, lib=L, p=0), types.SimpleNamespace(p=0)
    with pytest.raises(refusal or BonsaiError):
        Context.attn_insert(c, dims, b, b, b, 1, 0, b, b, b, b)
    with pytest.raises(refusal or BonsaiError):
        Context.attn_attend(c, dims, b, 0, b, None, b)


def test_number_follows_the_handle():
    """Objects whose handle was made elsewhere work, and a handle that is taken away is gone for every call."""
    build.build_lib()
    c, b = Context.__new__(Context), Buffer.__new__(Buffer)
    c.lib = lib.load_library()
    c.h, b.h = None, C.c_void_p(0x7000)
    assert (c.p, b.p) == (0, 0x7000) and b.h.value == 0x7000
    with pytest.raises(BonsaiError, match="null context"):
        c.gemv_q81(b, 16, 512, b, b)
    b.h = None
    assert b.p == 0
    b.h = C.c_void_p()
    b.h.value = 0x8000                                      # (as a call that takes C.byref(b.h) does)
    assert b.p == 0x8000


@pytest.mark.parametrize("name", CALLS)
def test_arguments_arrive_in_order_and_whole(name):
    """Each argument, at its parameter's full width, against a function of the binding's signature in the entry point's place."""
    build.build_lib()
    build.build_fastcall()
    L = lib.load_library()
    from bonsai_vk_b200 import _fastcall
    types_ = [t if t in (C.c_int, C.c_size_t) else C.c_void_p for t in L._bn_signatures[name][1]]
    sent = [-7 - i if t is C.c_int else (0x0123456789ABCD00 << 4) + i for i, t in enumerate(types_)]
    got = []
    stub = C.CFUNCTYPE(C.c_int, *types_)(lambda *a: got.extend(a) or -77)
    try:
        _fastcall.bind({n: (C.cast(stub, C.c_void_p).value, stub) for n in CALLS})
        assert getattr(_fastcall, name)(*sent) == -77 and got == sent
    finally:
        lib._call_layer(L, L._bn_signatures)


def test_call_layer_is_rebuilt_for_another_header(monkeypatch):
    """The layer's types are the header's: a changed header makes the built file stale."""
    seen = []
    monkeypatch.setattr(build, "_stale", lambda target, sources: seen.extend(sources))
    build.build_fastcall()
    assert any(s.endswith("bonsai_cuda.h") for s in seen)


def test_call_layer_is_named_for_its_interpreter():
    assert build.FASTCALL.endswith("_fastcall" + importlib.machinery.EXTENSION_SUFFIXES[0]) and "cpython" in build.FASTCALL


@pytest.mark.parametrize("failure", [OSError("no gcc"), types.SimpleNamespace(returncode=1, stdout="", stderr="Python.h: No such file")])
def test_build_goes_on_without_the_call_layer(monkeypatch, tmp_path, failure):
    def run(*a, **k):
        if isinstance(failure, OSError):
            raise failure
        return failure
    monkeypatch.setattr(build, "HERE", str(tmp_path))
    monkeypatch.setattr(build, "FASTCALL", str(tmp_path / "_fastcall.so"))
    (tmp_path / "_fastcall.so").write_bytes(b"an older one")
    monkeypatch.setattr(build.subprocess, "run", run)
    with pytest.warns(UserWarning, match="ctypes"):
        assert build.build_fastcall(force=True) is None
    assert not (tmp_path / "_fastcall.so").exists()
