"""Launches that ask for shared memory to spread their blocks, each as the first of its kernel: on a stand-in for the runtime, and on the
device in fresh processes."""
import ctypes as C
import itertools
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SMS = 148
# (static bytes, blocks per SM without more): the two-orientation MX cast's, and others
KERNELS = [(0, 8), (128, 8), (128, 32), (33792, 5)]
GRIDS = sorted({1, 16, 17} | {k * SMS + d for k in range(1, 9) for d in (0, 1)})


@pytest.fixture(scope="module")
def spread(tmp_path_factory):
    so = tmp_path_factory.mktemp("spread") / "spread.so"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic",  # its own stand-ins, not a CUDA runtime in this process
                           f"-I{ROOT / 'driss_torch_b200' / 'csrc'}", f"-I{cuda}/include", str(ROOT / "tests" / "spread_launch.cpp"), "-o", str(so)])
    lib = C.CDLL(str(so))
    first = itertools.product(range(64), range(64))  # a kernel on a device on which it never ran

    def call(grid, static, most, granted=1, on=None):
        which, dev = next(first) if on is None else on
        size, times, left = C.c_longlong(-1), C.c_int(-1), C.c_int(-1)
        e = lib.spread_launch(which, dev, C.c_uint(grid), C.c_longlong(static), most, granted, C.byref(size), C.byref(times), C.byref(left))
        return e, size.value, times.value, left.value, (which, dev)

    call.forget, call.move_to_green_context = lib.forget_what_was_allowed, lib.move_to_green_context
    return call


@pytest.mark.parametrize("static, most", KERNELS)
def test_the_first_launch_of_every_grid_is_taken(spread, static, most):
    for grid in GRIDS:
        error, size, times, left, _ = spread(grid, static, most)
        per_sm = 2 if grid <= 16 else -(-grid // SMS)
        assert (error, times, left) == (0, 1, 0), grid
        assert (size == 0) == (per_sm >= most), grid
        if size:  # its share of blocks fits an SM's 228 KB, with the kilobyte that each takes besides, and one more does not
            assert per_sm * (static + size + 1024) <= 228 * 1024 and (per_sm == 1 or (per_sm + 1) * (static + size + 1024) > 228 * 1024), grid


@pytest.mark.parametrize("static, most", KERNELS)
def test_no_more_is_asked_for_than_keeps_others_of_the_grid_off(spread, static, most):
    # what is left of an SM is for other kernels' blocks
    for grid in GRIDS:
        size, per_sm = spread(grid, static, most)[1], 2 if grid <= 16 else -(-grid // SMS)
        if size:
            assert (per_sm + 1) * (static + size + 1024 - 128) <= 228 * 1024 < (per_sm + 1) * (static + size + 1024), grid


@pytest.mark.parametrize("static, most", KERNELS)
def test_memory_that_is_not_granted_is_left_out(spread, static, most):
    for grid in GRIDS:
        assert spread(grid, static, most, granted=0)[:4] == (0, 0, 1, 0), grid


@pytest.mark.parametrize("static, most", KERNELS)
def test_a_grant_that_no_longer_holds_is_done_without(spread, static, most):
    error, size, times, left, on = spread(1, static, most)
    assert error == 0 and size > 0
    spread.forget()
    assert spread(1, static, most, on=on)[:4] == (0, 0, 1, 0)


@pytest.mark.parametrize("static, most", KERNELS)
def test_part_of_a_device_is_not_spread_over(spread, static, most):
    spread.move_to_green_context(1)
    try:
        for grid in GRIDS:
            assert spread(grid, static, most)[:4] == (0, 0, 1, 0), grid
    finally:
        spread.move_to_green_context(0)


_FIRST_CALL = """
import torch
import driss_torch_b200 as dt
tiles, call = {tiles}, {call!r}
a, s = dt.mx_fp8_quantize_blocked(torch.ones(256, 256, device="cuda").bfloat16())
dt.mx_fp8_bf16(a, a.t(), s, s)
x = (torch.randn(128, 128 * tiles, generator=torch.Generator("cuda").manual_seed(tiles), device="cuda") * 5).to(torch.bfloat16)
rows, columns = dt.mx_fp8_quantize(x), dt.mx_fp8_quantize(x.t().contiguous())
blocked = [dt.mx_fp8_quantize_blocked(x), dt.mx_fp8_quantize_blocked(x.t().contiguous())]
dt.mx_fp8_bf16(a, a.t(), s, s)  # the cast under test follows a product
got = {{"dual": lambda: dt.mx_fp8_quantize_dual(x), "dual blocked": lambda: dt.mx_fp8_quantize_dual(x, blocked=True),
       "transposed": lambda: dt.mx_fp8_quantize(x, transpose=True)}}[call]()
want = {{"dual": (*rows, *columns), "dual blocked": (*blocked[0], *blocked[1]), "transposed": columns}}[call]
assert len(got) == len(want) and all(torch.equal(g.contiguous().view(torch.uint8), w.view(torch.uint8)) for g, w in zip(got, want))
print("right")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["dual", "dual blocked", "transposed"])
@pytest.mark.parametrize("tiles", [2 * SMS + 1, 3 * SMS, 3 * SMS + 1, 4 * SMS])  # three and four blocks per SM, on either side of the step
def test_two_orientation_mx_cast_first_in_a_process(call, tiles):
    run = subprocess.run([sys.executable, "-c", _FIRST_CALL.format(tiles=tiles, call=call)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "right" in run.stdout, run.stderr[-2000:]


@pytest.mark.gpu
def test_two_orientation_mx_cast_in_a_green_context():
    import torch
    import driss_torch_b200 as dt
    from torch.cuda import green_contexts

    if not green_contexts.SUPPORTED:
        pytest.skip("torch without green contexts")
    x = torch.randn(1024, 2048, device="cuda").bfloat16()
    want = dt.mx_fp8_quantize_dual(x)
    torch.cuda.synchronize()
    part = green_contexts.GreenContext.create(32, torch.cuda.current_device())
    with torch.cuda.stream(part.Stream()):
        got = dt.mx_fp8_quantize_dual(x)
        torch.cuda.current_stream().synchronize()
    assert all(torch.equal(g.view(torch.uint8), w.view(torch.uint8)) for g, w in zip(got, want))
