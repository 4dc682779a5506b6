"""The wrappers' plain-function route to the operators: it answers, refuses and can be overridden as torch.ops does."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

import driss_torch_b200 as dt

E4M3 = torch.float8_e4m3fn


def calls(device):
    """Every wrapper with arguments that its operator accepts on a CUDA device (or a fake one)."""
    x = torch.randn(64, 128, device=device).to(torch.bfloat16)
    one = torch.ones(1, device=device)
    a = torch.zeros(64, 128, dtype=torch.uint8, device=device).view(E4M3)
    b = torch.zeros(32, 128, dtype=torch.uint8, device=device).view(E4M3).t()
    a4 = torch.zeros(64, 64, dtype=torch.uint8, device=device)
    b4 = torch.zeros(32, 64, dtype=torch.uint8, device=device).t()
    s = torch.full((512,), 127, dtype=torch.uint8, device=device).view(torch.float8_e8m0fnu)
    rows, cols = torch.ones(64, 1, device=device), torch.ones(1, 32, device=device)
    bias = torch.zeros(32, device=device)
    tune = (torch.bfloat16, False, 1, 1, 1, False, 1)
    return [
        ("saturated_cast", (x, one, E4M3, False)), ("saturated_cast_transposed", (x, one, E4M3)),
        ("saturated_cast_dual", (x, one, E4M3)), ("amax", (x,)), ("dynamic_scaled_quant", (x, E4M3)),
        ("dynamic_scaled_quant_with_scale", (x, E4M3)), ("dynamic_scaled_quant_rowwise", (x, E4M3)),
        ("dynamic_scaled_quant_dual", (x, E4M3)), ("cast_with_amax", (x, one, E4M3)), ("cast_with_amax_dual", (x, one, E4M3)),
        ("mx_fp8_quantize", (x, 32, 1, False, E4M3)), ("mx_fp8_quantize_with_amax", (x,)), ("mx_fp8_quantize_dual", (x, True)),
        ("mx_fp8_quantize_blocked", (x,)), ("mx_fp4_quantize", (x, True)), ("mx_fp8_bf16", (a, b, s, s)),
        ("mx_fp4_bf16", (a4, b4, s, s)), ("sweep_mm", (a, b, rows, cols, None, *tune)), ("sweep_mm", (a, b, rows, cols, bias, *tune)),
    ]


def outputs(r):
    return r if isinstance(r, tuple) else (r,)


def refusal(fn, args):
    with pytest.raises(Exception) as e:
        fn(*args)
    return type(e.value), str(e.value).splitlines()[0]


def test_every_wrapper_has_a_direct_call():
    names = {name for name, _ in calls("cpu")}
    assert names == {n for n in dir(dt.direct) if not n.startswith("_")}
    assert names | {"mx_cast", "check_device_status", "ShardedQuantizer"} == set(dt.__all__)


@pytest.mark.parametrize("i", range(19))
def test_no_cpu_kernel_and_signatures(i):
    # the first call of each also checks the C++ signature against the registration
    name, args = calls("cpu")[i]
    got = refusal(getattr(dt.direct, name), args)
    assert got[0] is NotImplementedError
    assert got == refusal(getattr(dt.ops, name), args)


@pytest.mark.parametrize("i", range(19))
def test_fake_tensors(i):
    with FakeTensorMode():
        name, args = calls("cuda")[i]
        got, want = outputs(getattr(dt, name)(*args)), outputs(getattr(dt.ops, name)(*args))
        assert [(g.shape, g.dtype, g.device, g.stride()) for g in got] == [(w.shape, w.dtype, w.device, w.stride()) for w in want]


X = torch.zeros(32, 32)


@pytest.mark.parametrize("name, args", [
    ("amax", ()), ("amax", (X, X)), ("amax", (None,)), ("amax", (1.0,)), ("dynamic_scaled_quant", (X, 3)),
    ("saturated_cast", (X, X, E4M3, 0)), ("saturated_cast", (X, X, E4M3, None)), ("mx_fp8_quantize", (X, 32.5, 1, False, E4M3)),
    ("mx_fp8_quantize", (X, 2 ** 70, 1, False, E4M3)), ("mx_fp8_quantize", (X, True, 1, False, E4M3)),
    ("sweep_mm", (X, X, X, X, 1, torch.bfloat16, False, 1, 1, 1, False, 1)),
])
def test_wrong_arguments_are_refused_alike(name, args):
    assert refusal(getattr(dt.direct, name), args) == refusal(getattr(dt.ops, name), args)


def test_torch_function_subclasses_and_modes():
    class Sub(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            return "subclass"

    class Mode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return "mode"

    assert dt.amax(X.as_subclass(Sub)) == "subclass"
    assert dt.saturated_cast(X, X.as_subclass(Sub), E4M3) == "subclass"
    with Mode():
        assert dt.amax(X) == "mode"


def test_calls_left_to_torch_ops_look_the_operator_up_once(monkeypatch):
    # a default device is such a mode: a program that sets one makes every call this way
    looked_up = []

    class Ops:  # torch looks the operator up itself under a mode: the wrappers add nothing to that
        def __getattr__(self, name):
            looked_up.append(name)
            return getattr(torch._ops.ops, name)

    def lookups(functions):
        looked_up.clear()
        with torch.device("meta"):
            shapes = [[o.shape for o in outputs(f(*args))] for f, (_, args) in zip(functions, calls("meta"))]
        return shapes, list(looked_up)

    names = [name for name, _ in calls("meta")]
    operators, wrappers = [getattr(dt.ops, n) for n in names], [getattr(dt.direct, n) for n in names]
    lookups(wrappers)
    monkeypatch.setattr(torch, "ops", Ops())
    assert lookups(wrappers) == lookups(operators)


def test_dispatch_modes_see_the_operator():
    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return torch.empty(1)

    with Mode():
        dt.amax(X)
    assert seen == ["DrissTorch.amax.default"]


def test_vmap_refuses_alike():
    y = torch.zeros(3, 4, 4)
    assert refusal(torch.vmap(dt.amax), (y,))[0] is refusal(torch.vmap(dt.ops.amax), (y,))[0]


@pytest.mark.parametrize("name", [n for n in dt.__all__ if n not in ("ShardedQuantizer", "check_device_status")])
def test_wrappers_can_be_scripted(name):
    graph = str(torch.jit.script(getattr(dt, name)).graph)
    assert "DrissTorch::" in graph


@pytest.mark.gpu
def test_same_results_as_torch_ops_and_under_tracing():
    for name, args in calls("cuda"):
        got, want = outputs(getattr(dt, name)(*args)), outputs(getattr(dt.ops, name)(*args))
        assert len(got) == len(want)
        for g, w in zip(got, want):
            assert (g.shape, g.dtype, g.stride()) == (w.shape, w.dtype, w.stride())
            assert torch.equal(g.contiguous().view(torch.uint8), w.contiguous().view(torch.uint8)), name
    x = torch.randn(64, 128, device="cuda").to(torch.bfloat16)
    traced = torch.jit.trace(dt.amax, (x,))
    assert "DrissTorch::amax" in str(traced.graph)
    y = x * 2
    assert torch.equal(traced(y), dt.amax(y))
