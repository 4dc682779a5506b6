"""Grids of less than a full wave ask for shared memory so that their blocks spread over the device (spread_bytes in dtq_host.h):
the same bytes, and a launch that the device takes, on either side of every step of that rule."""
import pytest
import torch

pytestmark = pytest.mark.gpu
E4M3, E5M2 = torch.float8_e4m3fn, torch.float8_e5m2
SMS = 148
# blocks: where the share per SM changes, from two for the smallest grids to as many as fit
GRIDS = [1, 16, 17, SMS, SMS + 1, 2 * SMS, 2 * SMS + 1, 5 * SMS, 5 * SMS + 1, 7 * SMS, 7 * SMS + 1, 8 * SMS + 1]


def _same(a, b):
    return torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))


@pytest.fixture(scope="module")
def x():
    return (torch.randn(max(GRIDS) * 8, 1024, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda") * 5).to(torch.bfloat16)


@pytest.mark.parametrize("name", ["mx", "mx_e5m2", "mx_fp32", "mx_fp4", "rowwise"])
def test_casts_of_every_share_per_sm(x, name):
    import driss_torch_b200 as dt

    op = {"mx": dt.mx_fp8_quantize, "mx_e5m2": lambda v: dt.mx_fp8_quantize(v, ScalarType=E5M2), "mx_fp32": lambda v: dt.mx_fp8_quantize(v.float()),
          "mx_fp4": dt.mx_fp4_quantize, "rowwise": lambda v: dt.dynamic_scaled_quant_rowwise(v, E4M3)}[name]
    rows_per_block = {"mx_fp32": 4, "rowwise": 8}.get(name, 8)  # 16 KB of input a block, or a row a warp
    whole = op(x)
    for grid in GRIDS:
        rows = grid * rows_per_block
        part = op(x[:rows])
        for p, w in zip(part, whole):
            n = p.numel()
            assert _same(p.flatten(), w.flatten()[:n]), (grid, rows)


@pytest.mark.parametrize("rows", [32 * 1, 32 * 17])  # a row of tiles, and five with a ragged last one
def test_two_orientation_mx_cast_of_every_share_per_sm(rows):
    import driss_torch_b200 as dt

    row_tiles = -(-rows // 128)
    for grid in (1, 16, 17, SMS, SMS + 1, 2 * SMS, 3 * SMS, 4 * SMS, 4 * SMS + 1, 5 * SMS + 1):
        cols = 128 * max(1, grid // row_tiles)
        v = (torch.randn(rows, cols, generator=torch.Generator(device="cuda").manual_seed(grid), device="cuda") * 5).to(torch.bfloat16)
        p, s, pt, st = dt.mx_fp8_quantize_dual(v)
        wp, ws = dt.mx_fp8_quantize(v)
        wpt, wst = dt.mx_fp8_quantize(v.t().contiguous())
        assert _same(p, wp) and _same(s, ws) and _same(pt, wpt) and _same(st, wst), grid
