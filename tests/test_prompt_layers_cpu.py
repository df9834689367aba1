"""The native launches of a prompt step (csrc/prompt_layers.cpp) with stand-ins for the launchers: a launch that fails ends
the step, is the one that is named, and leaves the library's math mode as it was."""

import ctypes

import pytest

from redline_b200.engine import prompt_layers as PL
from redline_b200.ops import build

LAYERS = 3


def calls_of(T, num_decode, failing=None, code=0):
    """(names of the launchers called, what the step returned, its counts); call number ``failing`` returns ``code``."""
    called, math = [], []

    def stand_in(name):
        def launch(*args):
            called.append(name)
            if name == "cublasSetMathMode":
                math.append(args[1])
            return code if len(called) - 1 == failing else 0
        kinds = [ctypes.c_void_p, ctypes.c_int] if name == "cublasSetMathMode" else []
        return ctypes.CFUNCTYPE(ctypes.c_int, *kinds)(launch)     # (the others: arguments are not looked at)

    fns = [stand_in(name) for name in PL._LAUNCHERS]
    layers = (PL._Layer * LAYERS)()
    plan = PL._Plan(*[ctypes.cast(f, ctypes.c_void_p).value for f in fns], ctypes.addressof(layers))
    plan.num_layers, plan.tc_min_rows = LAYERS, 128
    step = PL._Step()
    step.T, step.num_decode, step.num_tiles = T, num_decode, 1
    lib = ctypes.CDLL(build.compile_module("prompt_layers", "prompt_layers.cpp"))
    lib.rl_prompt_layers.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    n = PL._Counts()
    got = lib.rl_prompt_layers(ctypes.addressof(plan), ctypes.addressof(step), 1 if T <= 64 else 0, ctypes.addressof(n))
    assert math == [] if T <= 64 else math == ([16] if failing == 0 else [16, 0])
    return called, got, n


@pytest.mark.parametrize("T,num_decode", [(40, 0), (64, 3), (65, 0), (127, 1), (128, 0), (300, 2)])
def test_a_failed_launch_is_the_one_named(T, num_decode):
    called, got, n = calls_of(T, num_decode)
    many = T > 64
    attend = ["rope_kv_write"] + (["attn_decode"] if num_decode else []) + ["attn_prefill"]
    gate_up = ["gemm_tc"] if T >= 128 else ["cublasGemmEx", "swiglu"]
    layer = (["add_rmsnorm", "cublasGemmEx"] + attend + ["cublasGemmEx", "add_rmsnorm"] + gate_up + ["cublasGemmEx"] if many
             else ["gemm_mid"] + attend + ["gemm_mid"] * 3)
    assert called == ((["cublasSetMathMode"] if many else ["add_rmsnorm"]) + LAYERS * layer + (["cublasSetMathMode"] if many else []))
    assert got == 0 and n.launches == (0 if many else 1) + LAYERS * ((3 if many else 4) + 2 + (2 if num_decode else 0))
    for i, name in enumerate(called):
        some, got, n = calls_of(T, num_decode, failing=i, code=700 + i)
        assert got == 700 + i and PL._LAUNCHERS[n.failed] == name
        back = ["cublasSetMathMode"] if many and 0 < i < len(called) - 1 else []
        assert some == called[:i + 1] + back


def test_the_library_of_another_torch(monkeypatch):
    """The library is looked for by the CUDA version that torch was built for; one that is not there is told of."""
    asked = []

    def nothing(name, mode):
        asked.append(name)
        raise OSError(name)
    monkeypatch.setattr(PL.ctypes, "CDLL", nothing)
    monkeypatch.setattr(PL.torch.version, "cuda", "13.1")
    with pytest.warns(UserWarning, match="libcublas.so.13"):
        assert PL._library("cublasGemmEx") is None
    assert asked == ["libcublas.so.13"]
