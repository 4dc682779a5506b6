"""Casts on one stream while a product that holds every SM for long runs on another."""
import pytest
import torch

pytestmark = pytest.mark.gpu
E4M3, E5M2 = torch.float8_e4m3fn, torch.float8_e5m2


@pytest.mark.parametrize("rows, cols", [(8, 8192), (64, 8192), (1024, 4096)])
@pytest.mark.parametrize("name", ["mx", "mx_blocked", "mx_e5m2", "mx_fp4", "rowwise"])
def test_a_cast_runs_beside_a_product(name, rows, cols):
    import driss_torch_b200 as dt

    op = {"mx": dt.mx_fp8_quantize, "mx_blocked": dt.mx_fp8_quantize_blocked, "mx_e5m2": lambda v: dt.mx_fp8_quantize(v, ScalarType=E5M2),
          "mx_fp4": lambda v: dt.mx_fp4_quantize(v, blocked=True), "rowwise": lambda v: dt.dynamic_scaled_quant_rowwise(v, E4M3)}[name]
    # 16 tiles of 256 x 256 for each pair of SMs: all are held until shortly before the end, some 700 us
    a, sa = dt.mx_fp8_quantize_blocked(torch.ones(37 * 256, 16384, device="cuda").bfloat16())
    b, sb = dt.mx_fp8_quantize_blocked(torch.ones(8192, 16384, device="cuda").bfloat16())
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    early = 0.0
    for _ in range(10):  # the host may be late in launching the cast: the best of ten
        start, cast_end, product_end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        torch.cuda.synchronize()
        with torch.cuda.stream(main):
            dt.mx_fp8_bf16(a, b.t(), sa, sb)
            start.record()
            dt.mx_fp8_bf16(a, b.t(), sa, sb)
            product_end.record()
        start.synchronize()  # the second product runs
        with torch.cuda.stream(side):
            op(x)
            cast_end.record()
        torch.cuda.synchronize()
        early = max(early, cast_end.elapsed_time(product_end))
    assert early > 0.2, f"the cast ended {early:.3f} ms before the product"
