"""Kernels that ask for their first tiles ahead of their dependency, in some ranges of sizes: every output against the CPU oracle on
both sides of each edge, and on inputs that the kernel queued just before is still writing when they are asked for."""
import pytest
import torch

import driss_torch_b200 as dt
from conftest import as_bytes, assert_fp8_equal
from driss_torch_b200 import _cabi
from oracle import quant_oracle as qo

pytestmark = pytest.mark.gpu

E4M3, E5M2 = torch.float8_e4m3fn, torch.float8_e5m2
SCALE = 100.0
MIB = 1 << 20


def _input(size, dtype, ragged, seed):
    """Rows of 4096 columns, `size` bytes of them, and with `ragged` one row more and 32 columns more."""
    rows, cols = size // (4096 * dtype.itemsize) + ragged, 4096 + 32 * ragged
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(rows, cols, generator=g, device="cuda").to(dtype)


def _rows_of(blocked, rows, kblocks):
    """Row-major scales out of the blocked layout; everything else in it has to be zero."""
    flat = as_bytes(blocked).view(-1)
    places = torch.from_numpy(qo.blocked_scale_offsets(rows, kblocks)).view(-1).long()
    rest = flat.clone()
    rest[places] = 0
    assert not rest.any(), "padding of the blocked scales"
    return flat[places]


# Edges of asks_ahead and amax_ask_chunks (dtq_host.h); `ragged` lies just above the edge and has a partial last tile.
@pytest.mark.parametrize("ragged", [0, 1])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("mib", [2, 16, 20, 22, 28, 40, 48, 80, 128])
def test_every_output_at_the_edges(mib, dtype, ragged):
    x = _input(mib * MIB, dtype, ragged, mib)
    cpu, scale = x.cpu(), torch.full((1,), SCALE, device="cuda")
    rows, cols = x.shape
    assert torch.equal(dt.amax(x).cpu(), qo.amax(cpu))
    assert_fp8_equal(dt.saturated_cast(x, scale, E5M2), qo.saturated_cast(cpu, SCALE, E5M2), E5M2, "cast")
    payload, amax, inverse = dt.dynamic_scaled_quant_rowwise(x, E4M3)
    want = qo.dynamic_scaled_quant_rowwise(cpu, E4M3)
    assert_fp8_equal(payload, want[0], E4M3, "row-wise")
    assert torch.equal(amax.cpu(), want[1]) and torch.equal(inverse.cpu(), want[2])
    for elem in (E4M3, E5M2):
        payload, scales = dt.mx_fp8_quantize(x, ScalarType=elem)
        want = qo.mx_quantize(cpu, elem)
        assert_fp8_equal(payload, want[0], elem, f"mx {elem}")
        assert torch.equal(as_bytes(scales).view(-1), as_bytes(want[1]).view(-1)), f"mx {elem} scales"
        if elem == E4M3 and dtype == torch.bfloat16:
            payload, scales = dt.mx_fp8_quantize_blocked(x)
            assert_fp8_equal(payload, want[0], elem, "mx blocked")
            assert torch.equal(_rows_of(scales, rows, cols // 32), as_bytes(want[1]).view(-1)), "blocked scales"
    payload, scales = dt.mx_fp4_quantize(x, blocked=True)
    want = qo.mx_quantize(cpu, "e2m1")
    assert torch.equal(payload.view(torch.uint8).cpu(), want[0]), "mx4"
    assert torch.equal(_rows_of(scales, rows, cols // 32), as_bytes(want[1]).view(-1)), "mx4 scales"


CONSUMERS = {
    "amax": lambda y, s: (dt.amax(y),),
    "cast": lambda y, s: (dt.saturated_cast(y, s, E4M3),),
    "amax, both casts": lambda y, s: (dt.amax(y), *dt.saturated_cast_dual(y, s, E4M3)),
    "amax, cast": lambda y, s: (dt.amax(y), dt.saturated_cast(y, s, E4M3)),
    "mx": lambda y, s: dt.mx_fp8_quantize(y),
    "mx blocked": lambda y, s: dt.mx_fp8_quantize_blocked(y),
    "mx both": lambda y, s: dt.mx_fp8_quantize_dual(y, blocked=True),
    "mx e5m2": lambda y, s: dt.mx_fp8_quantize(y, ScalarType=E5M2),
    "mx4": lambda y, s: dt.mx_fp4_quantize(y, blocked=True),
    "rowwise": lambda y, s: dt.dynamic_scaled_quant_rowwise(y, E4M3),
    "tensorwise": lambda y, s: dt.dynamic_scaled_quant_with_scale(y, E4M3),
    "tensorwise both": lambda y, s: dt.dynamic_scaled_quant_dual(y, E4M3),
}


# Outputs of 0.5 MiB (a product that splits K; the tensor-wise quantization in one cluster), 2, 16, 24, 48 and 80 MiB.
@pytest.mark.parametrize("rows, n, k, kernel", [
    (64, 4096, 8192, "split"), (256, 4096, 512, "narrow"), (2048, 4096, 512, "pair"), (3072, 4096, 512, "wide"), (6144, 4096, 512, "pair"),
    (10240, 4096, 256, "pair"),
])
@pytest.mark.parametrize("name", CONSUMERS)
def test_input_that_the_product_before_still_writes(name, rows, n, k, kernel):
    # One buffer, written by products of two sets of operands in turn and read right behind each: a line that was asked for too
    # early and kept would be the other product's.
    g = torch.Generator(device="cuda").manual_seed(rows)
    scale = torch.full((1,), SCALE, device="cuda")
    weights, weight_scales = dt.mx_fp8_quantize_blocked(torch.randn(n, k, generator=g, device="cuda").to(torch.bfloat16))
    sets = [dt.mx_fp8_quantize_blocked((torch.randn(rows, k, generator=g, device="cuda") * f).to(torch.bfloat16)) for f in (1.0, 0.03)]
    y = torch.empty(rows, n, dtype=torch.bfloat16, device="cuda")

    def product(i):
        a, s = sets[i % 2]
        _cabi.mx_fp8_bf16(a, weights, s, weight_scales, out=y, kernel=kernel)

    want = []
    for i in range(2):
        product(i)
        torch.cuda.synchronize()
        want.append(CONSUMERS[name](y, scale))
        torch.cuda.synchronize()
    assert any(not torch.equal(as_bytes(a), as_bytes(b)) for a, b in zip(*want))
    got = []
    for i in range(6):
        product(i)
        got.append(CONSUMERS[name](y, scale))
    torch.cuda.synchronize()
    for i, outs in enumerate(got):
        assert all(torch.equal(as_bytes(a), as_bytes(b)) for a, b in zip(outs, want[i % 2])), i
