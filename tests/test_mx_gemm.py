"""mx_fp8_bf16: the MX block-scaled GEMM that consumes the MX casts.

CPU part: the oracle's restatement (oracle_mx_gemm_bf16) against an independent evaluation with
PyTorch CPU ops, its e4m3 / e8m0 decoders against PyTorch's casts, its blocked-scale indexing.
GPU part, modelled on the reference's test (test/test_mx.py:9-67): operands from the MX casts,
result against a bf16 matmul of the dequantised operands with the reference's own bar (SQNR above
80 dB) on the reference's size grid; and, because a tensor-core accumulation order cannot be
restated on a CPU, byte-exact equality with the oracle on inputs whose partial sums are all exactly
representable (small integers times powers of two), including shapes that are not multiples of the
tile and of the scale atoms.
"""
import pytest
import torch

from conftest import as_bytes
from oracle import quant_oracle as qo

E4M3 = torch.float8_e4m3fn
E8M0 = torch.float8_e8m0fnu

# test/test_mx.py:41-57 (M, K, N)
REFERENCE_SIZES = [(128, 128, 128), (256, 256, 256), (384, 384, 384), (512, 512, 512), (768, 768, 768),
                   (1024, 1024, 1024), (8192, 8192, 8192), (128, 256, 384), (256, 384, 512), (129, 256, 384),
                   (133, 512, 528)]


def _dequant(payload, scales_row_major, rows, k):
    s = torch.exp2(scales_row_major.view(torch.uint8).float() - 127.0).view(rows, k // 32, 1)
    return (payload.float().view(rows, k // 32, 32) * s).view(rows, k)


def _sqnr(want, got):
    # torchao.float8.float8_utils.compute_error as the reference's test uses it: 20 log10(|x| / |x - y|)
    err = (want.float() - got.float()).norm()
    return float("inf") if err == 0 else float(20 * torch.log10(want.float().norm() / err))


def _small_int_operands(m, n, k, seed):
    g = torch.Generator().manual_seed(seed)
    a = torch.randint(-3, 4, (m, k), generator=g).float().to(E4M3)
    b = torch.randint(-3, 4, (n, k), generator=g).float().to(E4M3)
    sa = torch.randint(125, 130, (m, k // 32), generator=g).to(torch.uint8)
    sb = torch.randint(125, 130, (n, k // 32), generator=g).to(torch.uint8)
    return a, b, sa, sb


_ORACLE_CACHE = {}


def _oracle_cached(a, b, sab, sbb, key):
    if key not in _ORACLE_CACHE:
        _ORACLE_CACHE[key] = qo.mx_gemm_bf16(a, b, sab, sbb)
    return _ORACLE_CACHE[key]


# ---- CPU: the oracle itself ----------------------------------------------------------------------------

def test_oracle_decoders_match_pytorch_casts():
    every = torch.arange(256, dtype=torch.int32).to(torch.uint8)
    every[0x7F] = 0  # the two NaN encodings would poison every sum (NaN x 0); checked on their own below
    every[0xFF] = 0
    a = every.view(E4M3).view(1, 256).repeat(8, 1)  # [8, 256]: every finite e4m3 byte as an A row
    ident = torch.zeros(256, 256)
    ident.fill_diagonal_(1.0)
    one_scales = torch.full((256 * 8,), 127, dtype=torch.uint8)
    sa = qo.to_blocked(one_scales[: 8 * 8], 8, 8)
    sb = qo.to_blocked(one_scales, 256, 8)
    out = qo.mx_gemm_bf16(a, ident.to(E4M3), sa, sb)  # picks out each element: bf16(e4m3 value), exact
    assert torch.equal(out[0].float(), every.view(E4M3).float())
    nan_row = torch.zeros(1, 32, dtype=torch.uint8)
    nan_row[0, 5] = 0x7F
    s1 = qo.to_blocked(torch.full((1,), 127, dtype=torch.uint8), 1, 1)
    assert qo.mx_gemm_bf16(nan_row.view(E4M3), torch.ones(1, 32).to(E4M3), s1, s1).float().isnan().all()
    # e8m0: 2^(b - 127); a single 1.0 x 1.0 product per output scaled by sa only
    for byte in (0, 1, 100, 127, 128, 200, 254):
        s = torch.full((4,), byte, dtype=torch.uint8)
        x = torch.zeros(1, 128)
        x[0, 0] = 1.0
        o = qo.mx_gemm_bf16(x.to(E4M3), x.to(E4M3), qo.to_blocked(s, 1, 4), qo.to_blocked(torch.full((4,), 127, dtype=torch.uint8), 1, 4))
        assert o.float().item() == 2.0 ** (byte - 127) or (byte < 127 - 126 - 7 and o.float().item() == 0.0)


@pytest.mark.parametrize("m,n,k", [(8, 16, 32), (33, 40, 96), (130, 136, 160), (64, 48, 512)])
def test_oracle_against_an_independent_evaluation(m, n, k):
    g = torch.Generator().manual_seed(m * 1000 + n)
    a = (torch.randn(m, k, generator=g) * 3).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g) * 0.1).to(torch.bfloat16)
    pa, sa = qo.mx_fp8_quantize(a)
    pb, sb = qo.mx_fp8_quantize(b)
    out = qo.mx_gemm_bf16(pa, pb, qo.to_blocked(sa, m, k // 32), qo.to_blocked(sb, n, k // 32))
    want = (_dequant(pa, sa, m, k).double() @ _dequant(pb, sb, n, k).double().t()).to(torch.bfloat16)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


# ---- GPU ----------------------------------------------------------------------------------------------------

@pytest.mark.gpu
@pytest.mark.parametrize("size", REFERENCE_SIZES, ids=lambda s: f"{s[0]}x{s[1]}x{s[2]}")
def test_reference_size_grid_sqnr(size):
    import driss_torch_b200 as dt

    m, k, n = size
    a = torch.rand(m, k, device="cuda").to(torch.bfloat16)
    b = torch.rand(n, k, device="cuda").to(torch.bfloat16)
    a_data, a_scale = dt.mx_fp8_quantize_blocked(a)
    b_data, b_scale = dt.mx_fp8_quantize_blocked(b)
    out = dt.mx_fp8_bf16(a_data, b_data.t(), a_scale, b_scale)
    assert out.shape == (m, n) and out.dtype == torch.bfloat16
    pa, sa = dt.mx_fp8_quantize(a)
    pb, sb = dt.mx_fp8_quantize(b)
    out_hp = _dequant(pa, sa, m, k).to(torch.bfloat16) @ _dequant(pb, sb, n, k).to(torch.bfloat16).t()
    assert _sqnr(out_hp, out) > 80, f"SQNR {_sqnr(out_hp, out)} dB"
    dt.check_device_status()


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["pair", "wide", "narrow"])
@pytest.mark.parametrize("m,n,k", [(128, 256, 128), (128, 128, 128), (256, 512, 512), (129, 256, 384), (133, 528, 512),
                                   (384, 384, 384), (64, 8, 32), (300, 520, 96), (1, 8, 64), (1024, 1024, 1024),
                                   (2560, 4096, 256),    # several rounds of tiles per SM: accumulator and stage reuse
                                   (18944, 504, 128),    # many tile rows, a ragged last tile column
                                   (9472, 376, 160)])    # a last tile column whose second scale atom does not exist
def test_exact_against_the_oracle_on_exactly_summable_inputs(m, n, k, kernel):
    # every kernel (an SM pair per 256 x 256 tile; one CTA per 128 x 256 or per 128 x 128 tile) on every size
    from driss_torch_b200 import _cabi

    a, b, sa, sb = _small_int_operands(m, n, k, seed=m + n + k)
    sab, sbb = qo.to_blocked(sa, m, k // 32), qo.to_blocked(sb, n, k // 32)
    want = _oracle_cached(a, b, sab, sbb, (m, n, k))
    out = _cabi.mx_fp8_bf16(a.cuda(), b.cuda(), sab.cuda(), sbb.cuda(), kernel=kernel)
    got = out.cpu()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16)), \
        f"{(got.view(torch.int16) != want.view(torch.int16)).sum().item()} of {got.numel()} outputs differ"
    assert _cabi.workspace_status(_cabi.workspace(torch.device("cuda", torch.cuda.current_device()))) == 0


@pytest.mark.gpu
def test_every_scale_position_is_used_where_it_belongs():
    # all data 1.0: out[m, n] = 32 * sum_kb 2^(sa[m,kb] + sb[n,kb] - 254); one k-block at a time carries a
    # row-dependent exponent, so a scale read from the wrong row, quadrant or k-block changes the result
    from driss_torch_b200 import _cabi

    m, n, k = 256, 512, 256
    ones_a = torch.ones(m, k).to(E4M3)
    ones_b = torch.ones(n, k).to(E4M3)
    for kb in range(k // 32):
        sa = torch.full((m, k // 32), 97, dtype=torch.uint8)
        sb = torch.full((n, k // 32), 97, dtype=torch.uint8)
        sa[:, kb] = (120 + torch.arange(m) % 13).to(torch.uint8)
        sb[:, kb] = (122 + torch.arange(n) % 11).to(torch.uint8)
        sab, sbb = qo.to_blocked(sa, m, k // 32), qo.to_blocked(sb, n, k // 32)
        want = qo.mx_gemm_bf16(ones_a, ones_b, sab, sbb)
        for kernel in ("pair", "wide", "narrow"):
            out = _cabi.mx_fp8_bf16(ones_a.cuda(), ones_b.cuda(), sab.cuda(), sbb.cuda(), kernel=kernel).cpu()
            assert torch.equal(out.view(torch.int16), want.view(torch.int16)), f"k-block {kb}, {kernel} kernel"


@pytest.mark.gpu
def test_operator_checks_fake_and_repeatability():
    import driss_torch_b200 as dt

    a = torch.rand(256, 512, device="cuda").to(torch.bfloat16)
    b = torch.rand(384, 512, device="cuda").to(torch.bfloat16)
    pa, sa = dt.mx_fp8_quantize_blocked(a)
    pb, sb = dt.mx_fp8_quantize_blocked(b)
    out = dt.mx_fp8_bf16(pa, pb.t(), sa, sb)
    for _ in range(3):  # the accumulation order is fixed: bit-identical from run to run
        assert torch.equal(as_bytes(dt.mx_fp8_bf16(pa, pb.t(), sa, sb).view(torch.int16)), as_bytes(out.view(torch.int16)))
    for bad in (
        lambda: dt.mx_fp8_bf16(pa, pb, sa, sb),                      # b must be the column-major [K, N] view
        lambda: dt.mx_fp8_bf16(pa, pb.t(), sa[:-1], sb),             # scale sizes as the reference's validate()
        lambda: dt.mx_fp8_bf16(pa, pb.t(), sa, sb[:-512]),
        lambda: dt.mx_fp8_bf16(pa.view(torch.uint8), pb.t(), sa, sb),
        lambda: dt.mx_fp8_bf16(pa[:, :96], pb.t(), sa, sb),
        lambda: dt.mx_fp8_bf16(pa, pb[:380].t(), sa, sb),            # N % 8
    ):
        with pytest.raises(RuntimeError):
            bad()
    with pytest.raises(NotImplementedError):
        dt.mx_fp8_bf16(pa.cpu(), pb.cpu().t(), sa.cpu(), sb.cpu())  # CUDA only
    torch._dynamo.reset()
    fn = torch.compile(dt.mx_fp8_bf16, fullgraph=True, backend="aot_eager")
    assert torch.equal(as_bytes(fn(pa, pb.t(), sa, sb).view(torch.int16)), as_bytes(out.view(torch.int16)))
    import driss_torch

    assert driss_torch.mx_fp8_bf16 is dt.mx_fp8_bf16
    dt.check_device_status()


# ---- MXFP4 (e2m1 packed two per byte): mx_fp4_bf16 -----------------------------------------------------------------

def test_oracle_fp4_against_an_independent_evaluation():
    g = torch.Generator().manual_seed(44)
    m, n, k = 40, 24, 192
    a = torch.randint(0, 256, (m, k // 2), generator=g).to(torch.uint8)
    b = torch.randint(0, 256, (n, k // 2), generator=g).to(torch.uint8)
    sa = torch.randint(120, 134, (m, k // 32), generator=g).to(torch.uint8)
    sb = torch.randint(120, 134, (n, k // 32), generator=g).to(torch.uint8)
    out = qo.mx_gemm_bf16(a, b, qo.to_blocked(sa, m, k // 32), qo.to_blocked(sb, n, k // 32), fp4=True)
    table = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0], dtype=torch.float64)

    def unpack(p, s, rows):
        lo, hi = table[(p & 0xF).long()], table[(p >> 4).long()]
        vals = torch.stack([lo, hi], dim=-1).view(rows, k)  # the lower index in the low nibble
        return (vals.view(rows, k // 32, 32) * torch.exp2(s.double() - 127).view(rows, k // 32, 1)).view(rows, k)

    want = (unpack(a, sa, m) @ unpack(b, sb, n).t()).to(torch.bfloat16)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16))


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["pair", "wide", "narrow"])
@pytest.mark.parametrize("m,n,k", [(128, 256, 256), (128, 128, 128), (256, 512, 1024), (129, 256, 384), (133, 528, 512),
                                   (64, 8, 32), (300, 520, 96), (1024, 1024, 1024), (2560, 2048, 512), (9472, 376, 320)])
def test_fp4_exact_against_the_oracle(m, n, k, kernel):
    # every product of two e2m1 values is a multiple of 1/4 below 64 and the scales span a few binades, so all
    # partial sums are exact in fp32 and the device must agree with the oracle bit for bit; K = 128, 384, 96, 320
    # leave the second scale atom of a 256-element stage partly or wholly outside the matrix
    from driss_torch_b200 import _cabi

    g = torch.Generator().manual_seed(m * 7 + n * 3 + k)
    a = torch.randint(0, 256, (m, k // 2), generator=g).to(torch.uint8)
    b = torch.randint(0, 256, (n, k // 2), generator=g).to(torch.uint8)
    sa = torch.randint(125, 130, (m, k // 32), generator=g).to(torch.uint8)
    sb = torch.randint(125, 130, (n, k // 32), generator=g).to(torch.uint8)
    sab, sbb = qo.to_blocked(sa, m, k // 32), qo.to_blocked(sb, n, k // 32)
    key = ("fp4", m, n, k)
    if key not in _ORACLE_CACHE:
        _ORACLE_CACHE[key] = qo.mx_gemm_bf16(a, b, sab, sbb, fp4=True)
    want = _ORACLE_CACHE[key]
    got = _cabi.mx_fp4_bf16(a.cuda(), b.cuda(), sab.cuda(), sbb.cuda(), kernel=kernel).cpu()
    assert torch.equal(got.view(torch.int16), want.view(torch.int16)), \
        f"{(got.view(torch.int16) != want.view(torch.int16)).sum().item()} of {got.numel()} outputs differ"
    assert _cabi.workspace_status(_cabi.workspace(torch.device("cuda", torch.cuda.current_device()))) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("size", REFERENCE_SIZES, ids=lambda s: f"{s[0]}x{s[1]}x{s[2]}")
def test_fp4_reference_size_grid_sqnr(size):
    # test/test_mx.py:36-67 with format "fp4": operands from the MXFP4 cast (scales straight in the blocked layout),
    # result against a bf16 matmul of the dequantised operands, SQNR above 80 dB
    import driss_torch_b200 as dt

    m, k, n = size
    a = torch.rand(m, k, device="cuda").to(torch.bfloat16)
    b = torch.rand(n, k, device="cuda").to(torch.bfloat16)
    a_data, a_scale = dt.mx_fp4_quantize(a, blocked=True)
    b_data, b_scale = dt.mx_fp4_quantize(b, blocked=True)
    out = dt.mx_fp4_bf16(a_data, b_data.t(), a_scale, b_scale)
    assert out.shape == (m, n) and out.dtype == torch.bfloat16
    table = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0], device="cuda")

    def dequant(x, rows):
        p, s = dt.mx_fp4_quantize(x)
        vals = torch.stack([table[(p & 0xF).long()], table[(p >> 4).long()]], dim=-1).view(rows, k)
        return (vals.view(rows, k // 32, 32) * torch.exp2(s.view(torch.uint8).float() - 127).view(rows, k // 32, 1)).view(rows, k)

    out_hp = dequant(a, m).to(torch.bfloat16) @ dequant(b, n).to(torch.bfloat16).t()
    assert _sqnr(out_hp, out) > 80, f"SQNR {_sqnr(out_hp, out)} dB"
    # the blocked scales are the row-major ones rearranged
    _, s_rm = dt.mx_fp4_quantize(a)
    assert torch.equal(as_bytes(a_scale), qo.to_blocked(s_rm.cpu(), m, k // 32))
    dt.check_device_status()


_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def _product(mode, operands, kernel):
    """One product through the C ABI, into an output with a poisoned margin on both sides."""
    from driss_torch_b200 import _cabi

    a, b, sa, sb, bias = operands
    m, n = a.shape[0], b.shape[0]
    room = torch.full((m * n + 128,), 0x5555, dtype=torch.int16, device="cuda")
    out = room[64:64 + m * n].view(torch.bfloat16).view(m, n)
    if mode == "rowwise":
        _cabi.rowwise_fp8_bf16(a, b, sa, sb, bias=bias, out=out, kernel=kernel)
    else:
        sab, sbb = (qo.to_blocked(s.cpu(), s.shape[0], s.shape[1]).cuda() for s in (sa, sb))
        (_cabi.mx_fp8_bf16 if mode == "mx8" else _cabi.mx_fp4_bf16)(a, b, sab, sbb, out=out, kernel=kernel)
    assert (room[:64] == 0x5555).all() and (room[64 + m * n:] == 0x5555).all(), "bytes outside the output were written"
    assert _cabi.workspace_status(_cabi.workspace(torch.device("cuda", torch.cuda.current_device()))) == 0
    return out


def _operands64(mode, operands):
    """The operands as fp64 matrices, block scales multiplied in."""
    a, b, sa, sb, _ = operands
    if mode == "rowwise":
        return a.double(), b.double()

    def full(v, s):
        if mode == "mx4":
            table = torch.tensor(_E2M1, dtype=torch.float64, device=v.device)
            v = torch.stack([table[(v & 0xF).long()], table[(v >> 4).long()]], dim=-1).view(v.shape[0], -1)
        scale = torch.where(s == 255, torch.full((), float("nan"), dtype=torch.float64, device=v.device), torch.exp2(s.double() - 127))
        return (v.double().view(v.shape[0], -1, 32) * scale.unsqueeze(2)).view(v.shape[0], -1)

    return full(a, sa), full(b, sb)


def _finish64(mode, operands, acc):
    if mode == "rowwise":
        acc = acc * operands[2].double()[:, None] * operands[3].double()[None, :]
        if operands[4] is not None:
            acc = acc + operands[4].double()
    return acc


def _check_exact_on_device(mode, m, n, k, kernel, a_dtype=E4M3, bias=None):
    # exactly summable inputs, so that fp64 on the device gives the same bits whatever the order of the sums
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randint(-3, 4, (m, k), generator=g, device="cuda").float()
    b = torch.randint(-3, 4, (n, k), generator=g, device="cuda").float()
    if mode == "rowwise":
        xs = torch.exp2(torch.randint(-3, 3, (m,), generator=g, device="cuda").float())
        ws = torch.exp2(torch.randint(-3, 3, (n,), generator=g, device="cuda").float())
        bias_d = None if bias is None else (torch.randint(-8, 9, (n,), generator=g, device="cuda") * 0.5).to(bias)
        operands = (a.to(a_dtype), b.to(E4M3), xs, ws, bias_d)
    else:
        sa = torch.randint(125, 130, (m, k // 32), generator=g, device="cuda").to(torch.uint8)
        sb = torch.randint(125, 130, (n, k // 32), generator=g, device="cuda").to(torch.uint8)
        if mode == "mx8":
            pa, pb = a.to(E4M3), b.to(E4M3)
        else:
            code = torch.tensor([13, 12, 10, 0, 2, 4, 5], dtype=torch.uint8, device="cuda")  # e2m1 of -3 .. 3
            pa, pb = (code[(v + 3).long()] for v in (a, b))
            pa, pb = pa[:, ::2] | (pa[:, 1::2] << 4), pb[:, ::2] | (pb[:, 1::2] << 4)
        operands = (pa, pb, sa, sb, None)
    got = _product(mode, operands, kernel)
    a64, b64 = _operands64(mode, operands)
    want = _finish64(mode, operands, a64 @ b64.t())
    assert torch.equal(got.view(torch.int16), want.to(torch.bfloat16).view(torch.int16))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "mx4", "rowwise"])
@pytest.mark.parametrize("m,n,k", [(4864, 4096, 160),   # 19 x 16 pair tiles: each accumulator used more than twice, 2 stages per tile
                                   (4700, 4104, 96)])   # the same with ragged last tiles and 16-byte stores
def test_pair_kernel_alternating_accumulators(m, n, k, mode):
    _check_exact_on_device(mode, m, n, k, "pair")


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "mx4", "rowwise"])
@pytest.mark.parametrize("tokens,n,kb", [(1, 8, 2048), (32, 136, 2064), (31, 9600, 4080),              # 32-token tiles, 2 CTAs per tile
                                         (33, 264, 4096), (64, 1000, 8192), (65, 520, 4208),           # 64 and 128 tokens, 4 to 8 CTAs
                                         (128, 4096, 8176), (129, 136, 8192), (300, 2056, 4096),       # several token tiles
                                         (16, 8192, 16384), (33, 264, 2048), (8, 19200, 4096)])        # the last two just outside the rule
def test_few_tiles_split_along_k(tokens, n, kb, mode):
    # `kb` bytes per operand row; K stages that do not divide evenly, a last stage that is partly past the end
    if mode != "rowwise":
        kb = kb // 32 * 32
    _check_exact_on_device(mode, tokens, n, kb * 2 if mode == "mx4" else kb, "auto",
                           a_dtype=torch.float8_e5m2 if tokens % 2 else E4M3, bias=[None, torch.float32, torch.bfloat16][tokens % 3])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "mx4", "rowwise"])
@pytest.mark.parametrize("kernel", ["pair", "wide", "narrow"])
@pytest.mark.parametrize("kb", [16, 32, 64, 80, 128, 144, 176, 224, 256, 2336])
def test_last_stage_takes_only_the_instructions_that_k_has(mode, kernel, kb):
    # bytes per operand row: one to four instructions of 32 in the last stage of 128, as the only stage and behind others;
    # 137 x 264: a ragged last tile both ways, and stores that end inside a chunk of 32 columns
    k = kb // 32 * 32 if mode == "mx8" else (kb * 2 if mode == "mx4" else kb)
    if k:
        _check_exact_on_device(mode, 137, 264, k, kernel, bias=torch.bfloat16 if kb % 64 else None)


# ---- the way out of a wait that runs out ---------------------------------------------------------------------------

def test_waits_of_the_gemm_roles_are_warp_wide():
    # What follows a role's wait is warp-wide (tcgen05.ld, elect.sync), and an abort flag raised between two lanes' polls
    # would split a warp that polls lane by lane.  So nothing but the two wrappers calls the per-thread wait.
    import re
    from pathlib import Path

    source = (Path(__file__).resolve().parents[1] / "driss_torch_b200" / "csrc" / "mx_gemm.cu").read_text()
    calls = re.findall(r"^.*\bmbar_wait\(.*$", source, flags=re.M)
    assert len(calls) == 3, calls  # its definition and the two wrappers
    # the same for the consumers of the TMA-staged MX cast: flag and barrier are looked at by vote
    staged = (Path(__file__).resolve().parents[1] / "driss_torch_b200" / "csrc" / "mx_cast_tma.cu").read_text()
    consumers = staged[staged.index("// consumers"):]
    assert "if (__any_sync(0xFFFFFFFFu, *static_cast<volatile int *>(&sm.abort) != 0)) return;" in consumers
    assert "if (!__all_sync(0xFFFFFFFFu, mbar_wait(&sm.full[s], round & 1u)))" in consumers
    # and the barrier that the way out waits for is committed to by nobody else
    assert len(re.findall(r"umma_commit\(&sm\.drained\)", source)) == len(re.findall(r"mbar_drain\(&sm\.drained", source)) == 2


def test_split_kernel_stores_only_if_no_cta_of_the_cluster_gave_up():
    # The abort flag is a CTA's own.  Every CTA adds up and stores all CTAs' partial sums of its tokens, so the flags of
    # all of them have to be asked for between the cluster barrier behind the partial sums and the stores.
    from pathlib import Path

    source = (Path(__file__).resolve().parents[1] / "driss_torch_b200" / "csrc" / "mx_gemm.cu").read_text()
    body = source[source.index("\nmx_gemm_split_kernel("):source.index("// ---- host side")]
    barrier, store = body.index("cluster_sync_all();"), body.index("stg_stream(p.out")
    assert "ld_cluster_u32(map_to_cta(smem_addr(&sm.abort), lane))" in body[barrier:store]
    assert "if (__any_sync(0xFFFFFFFFu, gave_up != 0)) break;" in body[barrier:store]


_WAIT_LIMIT_WORD = 40  # Workspace::wait_limit_us, csrc/dtq_host.h


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "rowwise"])
@pytest.mark.parametrize("kernel,m,n,k", [("pair", 256, 256, 1 << 18), ("wide", 256, 256, 1 << 18), ("narrow", 256, 256, 1 << 18),
                                          ("auto", 32, 128, 1 << 21)])  # split along K
def test_a_wait_that_runs_out_is_reported_and_stores_nothing(mode, kernel, m, n, k):
    # a sound launch whose epilogue waits hundreds of microseconds for its accumulator, under a limit of one
    from driss_torch_b200 import _cabi

    a, b = (torch.zeros(rows, k, dtype=torch.uint8, device="cuda").view(E4M3) for rows in (m, n))

    def run(ws):
        out = torch.full((m, n), 7.0, dtype=torch.bfloat16, device="cuda")
        if mode == "rowwise":
            _cabi.rowwise_fp8_bf16(a, b, torch.ones(m, device="cuda"), torch.ones(n, device="cuda"), out=out, ws=ws, kernel=kernel)
        else:
            sa, sb = (torch.full((_cabi.load().dtq_mx_gemm_scale_bytes(rows, k),), 127, dtype=torch.uint8, device="cuda") for rows in (m, n))
            _cabi.mx_fp8_bf16(a, b, sa, sb, out=out, ws=ws, kernel=kernel)
        return out

    ws = torch.zeros(_cabi.load().dtq_workspace_bytes(), dtype=torch.uint8, device="cuda")
    ws.view(torch.int32)[_WAIT_LIMIT_WORD] = 1
    out = run(ws)
    assert _cabi.workspace_status(ws) == 5  # DTQ_ERR_TIMEOUT
    assert (out == 7.0).all()
    ws = torch.zeros_like(ws)  # the context is as good as before
    assert (run(ws) == 0.0).all() and _cabi.workspace_status(ws) == 0


# ---- the kernel that splits K, by name ----------------------------------------------------------------------------

_SPLIT_SHAPES = [(1, 8, 2048), (32, 136, 2064), (31, 9600, 4080), (33, 264, 4096), (64, 1000, 8192), (65, 520, 4208),
                 (128, 4096, 8176), (129, 136, 8192), (300, 2056, 4096), (16, 8192, 16384)]  # tokens, outputs, bytes of K


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "mx4", "rowwise"])
@pytest.mark.parametrize("tokens,n,kb", _SPLIT_SHAPES + [(33, 264, 2048)])
def test_split_kernel_by_name_on_exactly_summable_inputs(tokens, n, kb, mode):
    if mode != "rowwise":
        kb = kb // 32 * 32
    _check_exact_on_device(mode, tokens, n, kb * 2 if mode == "mx4" else kb, "split",
                           a_dtype=torch.float8_e5m2 if tokens % 2 else E4M3, bias=[None, torch.float32, torch.bfloat16][tokens % 3])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "rowwise"])
def test_split_kernel_is_refused_where_there_is_nothing_to_split(mode):
    for tokens, n, kb in [(8, 19200, 4096), (8, 256, 1920)]:  # two CTAs for each of 150 tiles; 15 stages of K
        with pytest.raises(RuntimeError, match="unsupported shape"):
            _check_exact_on_device(mode, tokens, n, kb, "split")


def _random_operands(mode, m, n, kb, special=False):
    """Operands as the casts write them; ``special``: any byte as an element, and a few scales at either end."""
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n * 3 + kb)

    def rand_bytes(rows, cols, poison):
        v = torch.randint(0, 256, (rows, cols), generator=g, device="cuda", dtype=torch.int32).to(torch.uint8)
        # most rows free of NaN and infinity (e4m3 x1111111; e5m2 x11111yy), so that finite results are compared too
        return torch.where((v & 0x7C) == 0x7C, v & 0xBF, v) if not poison else torch.cat([v[:2], torch.where((v[2:] & 0x7C) == 0x7C, v[2:] & 0xBF, v[2:])])

    a_dtype = torch.float8_e5m2 if mode == "rowwise" else E4M3
    if mode == "mx4":
        a, b = (torch.randint(0, 256, (r, kb), generator=g, device="cuda", dtype=torch.int32).to(torch.uint8) for r in (m, n))
    elif special:
        a, b = rand_bytes(m, kb, True).view(a_dtype), rand_bytes(n, kb, True).view(E4M3)
    else:
        a = torch.randn(m, kb, generator=g, device="cuda").to(a_dtype)
        b = torch.randn(n, kb, generator=g, device="cuda").to(E4M3)
    if mode == "rowwise":
        return a, b, torch.rand(m, generator=g, device="cuda") + 0.5, torch.rand(n, generator=g, device="cuda") + 0.5, \
            torch.randn(n, generator=g, device="cuda")
    blocks = kb * (2 if mode == "mx4" else 1) // 32
    sa, sb = (torch.randint(118, 136, (r, blocks), generator=g, device="cuda", dtype=torch.int32).to(torch.uint8) for r in (m, n))
    if special:
        sa[m - 1, blocks - 1], sb[n - 1, 0], sb[n - 2, blocks // 2] = 255, 255, 0
        sa[0, 1] = 0
    return a, b, sa, sb, None


def _accumulation_bound(mode, operands, parts):
    """Largest distance of a correct result from the fp64 product: every step of 32 bytes of K and every part adds once
    in fp32 (an error below 2^-23 of the sum of magnitudes, truncation allowed), then one rounding to bf16, whose eight
    significant bits leave at most 2^-8 of the value."""
    a64, b64 = _operands64(mode, operands)
    steps = operands[0].shape[1] // 32 + parts + 4  # and the epilogue's three roundings
    want = _finish64(mode, operands, a64 @ b64.t())
    magnitude = _finish64(mode, operands[:4] + (None if operands[4] is None else operands[4].abs(),), a64.abs() @ b64.abs().t())
    slack = steps * 2.0**-23 * magnitude
    return want, slack + 2.0**-8 * (want.abs() + slack)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "mx4", "rowwise"])
@pytest.mark.parametrize("tokens,n,kb", _SPLIT_SHAPES)
def test_split_kernel_on_inexact_sums(tokens, n, kb, mode):
    if mode != "rowwise":
        kb = kb // 32 * 32
    operands = _random_operands(mode, tokens, n, kb)
    want, bound = _accumulation_bound(mode, operands, 8)
    split, straight, auto = (_product(mode, operands, kernel) for kernel in ("split", "narrow", "auto"))
    for got in (split, straight):
        assert ((got.double() - want).abs() <= bound).all()
    # further from fp64 than the straight sum by no more than chance (a handful of roundings in the smallest outputs)
    off = [float((got.double() - want).norm() / want.norm()) for got in (split, straight)]
    assert off[0] <= off[1] * (1.0 + 4.0 / want.numel() ** 0.5), off
    # and these shapes are what the default choice sends to this kernel
    assert torch.equal(auto.view(torch.int16), split.view(torch.int16))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mx8", "mx4", "rowwise"])
@pytest.mark.parametrize("tokens,n,kb", [(5, 256, 4096), (40, 136, 4096), (130, 264, 8192)])
def test_split_kernel_on_special_values(tokens, n, kb, mode):
    # NaN and (e5m2) infinite elements, scale bytes 0 and 255: what the straight sum makes of them, everywhere
    operands = _random_operands(mode, tokens, n, kb, special=True)
    split, straight = (_product(mode, operands, kernel) for kernel in ("split", "narrow"))
    assert torch.equal(split.isnan(), straight.isnan()) and torch.equal(split.isinf(), straight.isinf())
    assert torch.equal(split[split.isinf()], straight[split.isinf()])
    want, bound = _accumulation_bound(mode, operands, 8)
    finite = split.isfinite()
    assert finite.any() and not finite.all()
    assert ((split.double() - want).abs() <= bound)[finite].all()


# ---- the default choice (no device needed) -------------------------------------------------------------------------

def _choice(row_wise, m, n, k_bytes, sms=148, pairs=74, splits=1):
    from driss_torch_b200 import _cabi

    names = {code: name for name, code in _cabi.GEMM_KERNELS.items()}
    return names[_cabi.load().dtq_gemm_kernel_for(row_wise, m, n, k_bytes, sms, pairs, splits)]


@pytest.mark.parametrize("row_wise", [0, 1])
@pytest.mark.parametrize("tokens,n,kb", _SPLIT_SHAPES)
def test_choice_gives_way_where_clusters_cannot_be_launched(tokens, n, kb, row_wise):
    assert _choice(row_wise, tokens, n, kb) == "split"
    assert _choice(row_wise, tokens, n, kb, splits=0) in ("pair", "wide", "narrow")
    assert _choice(row_wise, tokens, n, kb, pairs=0, splits=0) in ("wide", "narrow")


def test_choice_at_the_edges_of_the_split_rule():
    for row_wise in (0, 1):
        # up to 32 tokens from the sixteenth stage of 128 bytes, up to 64 and above from the thirty-second
        for tokens, last_without in [(1, 1920), (32, 1920), (33, 3968), (64, 3968), (65, 3968), (300, 3968)]:
            assert _choice(row_wise, tokens, 1024, last_without) != "split", (tokens, last_without)
            assert _choice(row_wise, tokens, 1024, last_without + 1) == "split", (tokens, last_without)
        # two CTAs per tile (75 to 148 tiles) pay for 64 tokens, not for 128
        assert _choice(row_wise, 64, 148 * 128, 8192) == "split" and _choice(row_wise, 64, 149 * 128, 8192) != "split"
        assert _choice(row_wise, 128, 74 * 128, 8192) == "split" and _choice(row_wise, 128, 75 * 128, 8192) != "split"


def test_choice_leaves_the_reference_sizes_on_the_straight_sum():
    for m, k, n in REFERENCE_SIZES + [(4096, 4096, 4096), (2048, 1024, 8192)]:
        for k_bytes in (k, k // 2):
            assert _choice(0, m, n, k_bytes) != "split"


# (row-wise, tokens, outputs, bytes of K): the kernel that was the quickest of the three on a B200, by 3 to 30 %
_QUICKEST = [(0, 7666, 4840, 512, "wide"), (0, 6311, 8264, 320, "wide"), (0, 23978, 2424, 352, "wide"), (0, 25579, 2912, 192, "wide"),
             (0, 16182, 6256, 224, "wide"), (0, 677, 6608, 1072, "pair"), (0, 23290, 656, 1552, "pair"), (0, 8498, 256, 7040, "narrow"),
             (0, 3327, 376, 4704, "narrow"), (1, 3124, 12456, 1504, "pair"), (1, 17010, 744, 3040, "pair"), (1, 10367, 10248, 1008, "pair"),
             (1, 6629, 12728, 736, "pair")]


@pytest.mark.parametrize("row_wise,tokens,n,kb,quickest", _QUICKEST)
def test_choice_where_one_kernel_is_clearly_the_quickest(row_wise, tokens, n, kb, quickest):
    assert _choice(row_wise, tokens, n, kb) == quickest
