"""The casts ask for their first tiles ahead of their dependency in some ranges of sizes: same bytes on both sides of each edge,
checked against the same operator on slices of rows, which fall into another range."""
import pytest
import torch

import driss_torch_b200 as dt

pytestmark = pytest.mark.gpu

E4M3, E5M2 = torch.float8_e4m3fn, torch.float8_e5m2
OPS = {
    "cast": lambda x, s: dt.saturated_cast(x, s, E5M2),
    "mx": lambda x, s: dt.mx_fp8_quantize(x)[0],
    "mx e5m2": lambda x, s: dt.mx_fp8_quantize(x, ScalarType=E5M2)[0],
    "mx blocked": lambda x, s: dt.mx_fp8_quantize_blocked(x)[0],
    "mx4 blocked": lambda x, s: dt.mx_fp4_quantize(x, blocked=True)[0],
    "rowwise": lambda x, s: dt.dynamic_scaled_quant_rowwise(x, E4M3)[0],
}
# rows x columns of bf16 around 512 KiB, 16 MiB and 128 MiB, whole tiles and ragged ones
SHAPES = [(1, 32), (3, 96), (64, 4096), (65, 4064), (2047, 4096), (2048, 4096), (2051, 4128), (8191, 8192), (8192, 8192), (8193, 8192)]


@pytest.mark.parametrize("rows,cols", SHAPES)
def test_same_bytes_on_both_sides_of_the_edges(rows, cols):
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, cols, generator=g, device="cuda").to(torch.bfloat16)
    scale = torch.full((1,), 100.0, device="cuda")
    step = max(1, rows // 3 + 1)
    for name, op in OPS.items():
        whole = op(x, scale).view(torch.uint8)
        # slices as tensors of their own: 16-byte aligned, other sizes
        parts = [op(x[r:r + step].clone(), scale).view(torch.uint8) for r in range(0, rows, step)]
        assert torch.equal(whole, torch.cat(parts)), name
    assert torch.equal(dt.amax(x), x.abs().max().float().reshape(1))
