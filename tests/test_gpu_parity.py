"""Parity of the CUDA path (through the C ABI) with the CPU oracle on identical seeded inputs.

Bars: int8 codes, fp32 scales, int32 accumulators and all index work bit-exact; 16-bit outputs within
max-rel-err 1e-2 of the exact dequantised math (fp64), where
    rel = |y - ref| / max(|ref|, 1e-3 * max|ref|).
"""
import numpy as np
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

from conftest import from_bf16_bits
from oracle import oracle
from pyraquant_b200 import _lib, int8_exec, ops, routing

pytestmark = pytest.mark.gpu
TOL = 1e-2


def max_rel_err(y: torch.Tensor, ref64: torch.Tensor) -> float:
    ref = ref64.double()
    denom = torch.maximum(ref.abs(), 1e-3 * ref.abs().max())
    return float(((y.double() - ref).abs() / denom).max())


@pytest.fixture(autouse=True)
def _status_clean(cuda_dev):
    yield
    ops.check_device_status(cuda_dev)


def rand_act(M, K, dtype, seed, outliers=True):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(M, K, generator=g)
    if outliers and K >= 16:
        x[:, torch.randperm(K, generator=g)[: max(1, K // 200)]] *= 20.0
    return x.to(dtype)


# ------------------------------------------------------------------------------------------------ quantisation
@pytest.mark.parametrize("M,K", [(1, 64), (8, 64), (17, 640), (154, 1280), (513, 2048), (4350, 3072),
                                 (300, 5120), (200, 10240), (130, 12288), (96, 15360), (5, 20480), (33, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quant_rows_bit_exact(cuda_dev, M, K, dtype):
    x = rand_act(M, K, dtype, 100 + M + K)
    if M > 3:
        x[2].zero_()                          # all-zero token -> 1e-8 floor
        x[3] = x[3].abs().max()               # constant row: every code is 127
    q, s = int8_exec.quant_rows(x.to(cuda_dev))
    qo, so = oracle.quant_rows(x)
    assert q.dtype == torch.int8 and s.dtype == torch.float32 and q.shape == (M, K) and s.shape == (M,)
    assert torch.equal(s.cpu(), so)
    assert torch.equal(q.cpu(), qo)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quant_codes_at_rounding_ties(cuda_dev, dtype):
    """One row per significand of the absmax, holding every value of the nine binades below it (for fp16 every fourth
    significand and the exact half): the quotients that are rounding ties (absmax / 2 in every row, more where the
    significand is a multiple of 127) and all their neighbours get the codes of the IEEE division."""
    one, per = (0x3F80, 128) if dtype == torch.bfloat16 else (0x3C00, 1024)
    amax = torch.arange(one, one + per, 1 if per == 128 else 4, dtype=torch.int32)
    below = torch.arange(0, 9 * per, 1 if per == 128 else 4, dtype=torch.int32)
    bits = torch.cat([amax[:, None], amax[:, None] - per, (amax[:, None] - below[None, :])], dim=1)
    bits[:, 2::2] |= 0x8000                                          # alternate signs
    bits = torch.nn.functional.pad(bits, (0, (-bits.shape[1]) % 16))
    x = torch.where(bits >= 0x8000, bits - 0x10000, bits).to(torch.int16).view(dtype)
    q, s = int8_exec.quant_rows(x.to(cuda_dev))
    qo, so = oracle.quant_rows(x)
    assert torch.equal(s.cpu(), so) and torch.equal(q.cpu(), qo)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quant_scales_for_every_absmax(cuda_dev, dtype):
    """Every positive finite value of the activation type as a row's absmax: the scale equals the IEEE quotient
    absmax / 127 bit for bit (the kernel computes it with a multiply-and-correct sequence), and so do the group scales."""
    top = 0x7F80 if dtype == torch.bfloat16 else 0x7C00
    bits = torch.arange(1, top, dtype=torch.int32).to(torch.int16)
    vals = bits.view(dtype)
    M = vals.numel()
    x = torch.zeros(M, 32, dtype=dtype)
    x[:, 5] = vals
    x[::2, 17] = -vals[::2]
    _q, s = int8_exec.quant_rows(x.to(cuda_dev))
    want = vals.float().clamp_min(1e-8) / torch.full((M,), 127.0)
    assert torch.equal(s.cpu(), want)
    _q, sg = int8_exec.quant_rows_g32(x.to(cuda_dev))
    assert torch.equal(sg.cpu()[:, 0], want)


def test_quant_rows_cfg0_full(cuda_dev):
    L = oracle.make_layer(0, 4608, 3072, 8, lowrank=False, bias=False)
    q, s = int8_exec.quant_rows(L["x"].to(cuda_dev))
    qo, so = oracle.quant_rows(L["x"])
    assert torch.equal(s.cpu(), so) and torch.equal(q.cpu(), qo)


def test_quant_rows_strided_rows_and_views(cuda_dev):
    x = rand_act(64, 3072 + 1024, torch.bfloat16, 7).to(cuda_dev)
    view = x[:, 1024:]                                    # row stride 4096, offset 2048 bytes
    q, s = int8_exec.quant_rows(view)
    qo, so = oracle.quant_rows(view.cpu())
    assert torch.equal(q.cpu(), qo) and torch.equal(s.cpu(), so)
    odd = x[:, 3:3 + 64]                                  # misaligned start: falls back to a copy, same result
    q2, s2 = int8_exec.quant_rows(odd)
    qo2, so2 = oracle.quant_rows(odd.cpu())
    assert torch.equal(q2.cpu(), qo2) and torch.equal(s2.cpu(), so2)
    tr = x[:32, :32].t()                                  # last dim not contiguous
    q3, _ = int8_exec.quant_rows(tr)
    assert torch.equal(q3.cpu(), oracle.quant_rows(tr.cpu())[0])


def test_quant_rows_empty(cuda_dev):
    q, s = int8_exec.quant_rows(torch.empty(0, 64, dtype=torch.bfloat16, device=cuda_dev))
    assert q.shape == (0, 64) and s.shape == (0,)


def test_quant_rows_ties_exact(cuda_dev):
    # rows built so that many quotients land exactly on or next to .5: amax = 127 * 2^e makes scale a power of two
    base = torch.arange(-254, 255, dtype=torch.float32) * 0.5            # includes every k + 0.5
    rows = []
    for e in (-3, 0, 2):
        r = base * 2.0 ** e
        r = torch.cat([r, torch.tensor([127.0 * 2.0 ** e])])
        rows.append(torch.nn.functional.pad(r, (0, 512 - r.numel())))
    x = torch.stack(rows).to(torch.bfloat16)
    q, s = int8_exec.quant_rows(x.to(cuda_dev))
    qo, so = oracle.quant_rows(x)
    assert torch.equal(q.cpu(), qo) and torch.equal(s.cpu(), so)


@pytest.mark.parametrize("M,K", [(9, 64), (300, 640), (257, 1280), (64, 5120), (31, 2560)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quant_rows_g32_bit_exact(cuda_dev, M, K, dtype):
    x = rand_act(M, K, dtype, 200 + M + K)
    x[0, :32] = 0
    q, s = int8_exec.quant_rows_g32(x.to(cuda_dev))
    qo, so = oracle.quant_rows_g32(x)
    assert s.shape == (M, K // 32)
    assert torch.equal(s.cpu(), so) and torch.equal(q.cpu(), qo)


def test_gather_quant_rows_bit_exact(cuda_dev):
    canvas = rand_act(1024, 3072, torch.bfloat16, 11)
    g = torch.Generator().manual_seed(5)
    idx = torch.randint(0, 1024, (777,), generator=g, dtype=torch.int32)
    idx[5] = -1; idx[100] = -1; idx[776] = 1023; idx[0] = 0
    q, s = int8_exec.gather_quant_rows(canvas.to(cuda_dev), idx.to(cuda_dev))
    src = canvas[idx.clamp_min(0).long()].clone()
    src[idx < 0] = 0
    qo, so = oracle.quant_rows(src)
    assert torch.equal(q.cpu(), qo) and torch.equal(s.cpu(), so)
    plain = torch.ops.pq_b200.gather_rows(canvas.to(cuda_dev), idx.to(cuda_dev))
    assert torch.equal(plain.cpu(), src)


# ------------------------------------------------------------------------------------------------ GEMM
def run_gemm_case(dev, M, N, K, *, lowrank, bias, dtype=torch.bfloat16, seed=0, extreme=False):
    g = torch.Generator().manual_seed(seed)
    if extreme:
        xq = torch.full((M, K), 127, dtype=torch.int8); xq[::2] = -127
        wq = torch.full((N, K), 127, dtype=torch.int8); wq[1::3] = -127
    else:
        xq = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8)
        wq = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8)
    sr = torch.rand(M, generator=g) * 0.05 + 0.001
    sc = torch.rand(N, generator=g) * 0.002 + 0.0001
    b = torch.randn(N, generator=g) * 0.01 if bias else None
    t = lb = None
    if lowrank:
        t = (torch.randn(M, 32, generator=g) * 1.0).to(dtype)
        lb = (torch.randn(32, N, generator=g) * 0.02).to(dtype)
    to = lambda v: None if v is None else v.to(dev)
    out, acc = ops.int8_gemm_debug(to(xq), to(sr), to(wq), to(sc), to(b), to(t), to(lb), dtype)
    torch.cuda.synchronize()
    acc_ref = oracle.int_mm(xq, wq)
    assert torch.equal(acc.cpu(), acc_ref), f"int32 accumulators differ at {(acc.cpu() != acc_ref).sum().item()} places"
    ref64 = oracle.exact_dequant_f64(acc_ref, sr, sc, b, t, lb)
    err = max_rel_err(out.cpu(), ref64)
    assert err <= TOL, err
    # against the fp32 restatement of the kernel's epilogue: identical bits without the low-rank term (same
    # operations in the same order), summation-order noise of the rank-32 dot product with it
    y32 = oracle.epilogue(acc_ref, sr, sc, b, t, lb, dtype)
    if not lowrank:
        assert torch.equal(out.cpu(), y32)
    else:
        assert max_rel_err(out.cpu(), y32.double()) <= 8e-3
    return out


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (1, 256, 64), (8, 128, 64), (17, 384, 192), (154, 640, 640),
                                   (300, 512, 1280), (1000, 3072, 512), (257, 1280, 2560), (129, 264, 80),
                                   (4350, 1288, 144)])
def test_gemm_small_shapes(cuda_dev, M, N, K):
    run_gemm_case(cuda_dev, M, N, K, lowrank=True, bias=True, seed=M + N + K)        # low-rank term on tcgen05
    run_gemm_case(cuda_dev, M, N, K, lowrank=False, bias=False, seed=M + N + K + 1)
    ops.LOWRANK_ON_TENSOR_CORES = False                                             # low-rank term by mma.sync
    try:
        run_gemm_case(cuda_dev, M, N, K, lowrank=True, bias=True, seed=M + N + K)
    finally:
        ops.LOWRANK_ON_TENSOR_CORES = True


def test_gemm_extreme_accumulators_exact(cuda_dev):
    # |acc| = K * 127^2 = 2.0e8 > 2^24: only true int32 accumulation gets this right
    run_gemm_case(cuda_dev, 256, 512, 12288, lowrank=False, bias=True, extreme=True)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lowrank,bias", [(True, True), (True, False), (False, True)])
def test_gemm_dtypes_and_options(cuda_dev, dtype, lowrank, bias):
    run_gemm_case(cuda_dev, 777, 768, 1024, lowrank=lowrank, bias=bias, dtype=dtype, seed=3)


@pytest.mark.parametrize("bn,stages", [(128, 2), (128, 4), (128, 6), (256, 2), (256, 3), (256, 4)])
def test_gemm_tile_variants(cuda_dev, bn, stages):
    _lib.set_option("gemm_block_n", bn); _lib.set_option("gemm_stages", stages)
    try:
        run_gemm_case(cuda_dev, 1500, 1024, 768, lowrank=True, bias=True, seed=bn + stages)
    finally:
        _lib.set_option("gemm_block_n", 0); _lib.set_option("gemm_stages", 0)


def test_gemm_persistent_many_tiles_per_cta(cuda_dev):
    # few CTAs, many tiles each: exercises the accumulator double buffer and barrier phases
    _lib.set_option("gemm_max_ctas", 3)
    try:
        run_gemm_case(cuda_dev, 2000, 2048, 384, lowrank=True, bias=True, seed=9)
    finally:
        _lib.set_option("gemm_max_ctas", 0)


@pytest.mark.parametrize("pm,pn", [(1, 1), (2, 3), (5, 2), (16, 8)])
def test_gemm_schedule_grids(cuda_dev, pm, pn):
    # ragged CTA grids over the tile matrix: idle steps, column tile changes, both accumulator buffers
    _lib.set_option("gemm_pn", pn); _lib.set_option("gemm_pm", pm)
    try:
        run_gemm_case(cuda_dev, 1700, 2304, 256, lowrank=True, bias=True, seed=pm * 10 + pn)
    finally:
        _lib.set_option("gemm_pn", 0); _lib.set_option("gemm_pm", 0)


@pytest.mark.parametrize("M,N,K", [(256, 256, 128), (128, 256, 256), (300, 512, 192), (1000, 768, 640), (2049, 1288, 384),
                                   (4608, 3072, 3072)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("ew", [8, 16])
def test_gemm_cta_pair_kernel(cuda_dev, M, N, K, dtype, ew):
    """The cta_group::2 kernel forced on for every shape it accepts: odd numbers of 128-row tiles (one CTA of the
    last pair has no rows), ragged N, several tiles per pair, with and without the low-rank term; both epilogue
    widths (eight warps: long K; sixteen warps: short K) at every shape.  This is the accumulator-dumping instantiation, which
    stores from registers; the staged store is compared in test_gemm_staged_store_over_many_tiles."""
    _lib.set_option("gemm_pair", 2); _lib.set_option("gemm_epi_warps", ew)
    try:
        run_gemm_case(cuda_dev, M, N, K, lowrank=True, bias=True, dtype=dtype, seed=M + N)
        run_gemm_case(cuda_dev, M, N, K, lowrank=False, bias=True, dtype=dtype, seed=M + N + 1)
        _lib.set_option("gemm_max_ctas", 4)          # two pairs only: long per-pair tile sequences
        run_gemm_case(cuda_dev, M, N, K, lowrank=True, bias=False, dtype=dtype, seed=M + N + 2)
        run_gemm_case(cuda_dev, M, N, K, lowrank=False, bias=False, dtype=dtype, seed=M + N + 3)
    finally:
        _lib.set_option("gemm_pair", 1); _lib.set_option("gemm_max_ctas", 0); _lib.set_option("gemm_epi_warps", 0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_production_kernels_bit_equal_without_lowrank(cuda_dev, dtype):
    """The non-debug instantiations (what users run) against the fp32 restatement, no low-rank term: identical bits
    from every kernel variant."""
    g = torch.Generator().manual_seed(77)
    M, N, K = 900, 768, 384
    xq = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8)
    wq = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8)
    sr = torch.rand(M, generator=g) * 0.05 + 0.001
    sc = torch.rand(N, generator=g) * 0.002 + 0.0001
    b = torch.randn(N, generator=g) * 0.01
    y32 = oracle.epilogue(oracle.int_mm(xq, wq), sr, sc, b, None, None, dtype)
    d = cuda_dev
    for pair, bn, ew in ((0, 256, 0), (0, 128, 0), (2, 0, 8), (2, 0, 16)):
        _lib.set_option("gemm_pair", pair); _lib.set_option("gemm_block_n", bn); _lib.set_option("gemm_epi_warps", ew)
        try:
            y = int8_exec.int8_gemm_fused(xq.to(d), sr.to(d), wq.to(d), sc.to(d), b.to(d), dtype)
        finally:
            _lib.set_option("gemm_pair", 1); _lib.set_option("gemm_block_n", 0); _lib.set_option("gemm_epi_warps", 0)
        assert torch.equal(y.cpu(), y32), (pair, bn, ew)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,ew,pair", [(8192, 1288, 320, 16, 2), (3001, 2376, 1808, 0, 1), (30000, 320, 320, 0, 1), (257, 136, 128, 16, 2),
                                           (2048, 1032, 2304, 8, 2)])
def test_gemm_pair_epilogues_bit_equal_on_many_outputs(cuda_dev, dtype, M, N, K, ew, pair):
    """Product and sum of the epilogue are rounded separately: a fused multiply-add shows in about one output of 100 000, so
    millions of outputs are compared with torch's separate fp32 operations (the accumulators are exact in fp64 and below
    2^24).  Ragged row and column tails of the tiles that leave through shared memory, and the choice of kernel by size."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    xq = torch.randint(-127, 128, (M, K), generator=g, device=cuda_dev, dtype=torch.int8)
    wq = torch.randint(-127, 128, (N, K), generator=g, device=cuda_dev, dtype=torch.int8)
    sr = torch.rand(M, generator=g, device=cuda_dev) * 0.05 + 0.001
    sc = torch.rand(N, generator=g, device=cuda_dev) * 2e-4 + 1e-5
    b = torch.randn(N, generator=g, device=cuda_dev) * 0.01
    acc = (xq.double() @ wq.double().t())
    assert acc.abs().max().item() < 2 ** 24
    want = ((acc.float() * (sr[:, None] * sc[None, :])) + b[None, :]).to(dtype)
    _lib.set_option("gemm_pair", pair); _lib.set_option("gemm_epi_warps", ew)
    try:
        y = int8_exec.int8_gemm_fused(xq, sr, wq, sc, b, dtype)
    finally:
        _lib.set_option("gemm_pair", 1); _lib.set_option("gemm_epi_warps", 0)
    assert torch.equal(y, want)


def _exact_gemm_operands(cuda_dev, M, N, K, dtype):
    """Operands whose accumulators are exact in fp64 and below 2^24, and the output of torch's separate fp32 operations."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    xq = torch.randint(-127, 128, (M, K), generator=g, device=cuda_dev, dtype=torch.int8)
    wq = torch.randint(-127, 128, (N, K), generator=g, device=cuda_dev, dtype=torch.int8)
    sr = torch.rand(M, generator=g, device=cuda_dev) * 0.05 + 0.001
    sc = torch.rand(N, generator=g, device=cuda_dev) * 2e-4 + 1e-5
    b = torch.randn(N, generator=g, device=cuda_dev) * 0.01
    acc = xq.double() @ wq.double().t()
    assert acc.abs().max().item() < 2 ** 24
    return xq, wq, sr, sc, b, ((acc.float() * (sr[:, None] * sc[None, :])) + b[None, :]).to(dtype)


@pytest.fixture
def gemm_options():
    """Sets library options for one test and puts the defaults back."""
    defaults = {"gemm_pair": 1, "gemm_block_n": 0, "gemm_epi_warps": 0, "gemm_tma_store": 1, "gemm_max_ctas": 0}

    def set_options(**kw):
        for k, v in {**defaults, **kw}.items():
            _lib.set_option(k, v)
    yield set_options
    set_options()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(2049, 1280, 128), (1500, 1032, 1296), (700, 264, 640)])
def test_gemm_staged_store_over_many_tiles(cuda_dev, gemm_options, dtype, M, N, K):
    """Sixteen-warp tiles that leave through shared memory, in the kernel users run: two SM pairs go through all tiles, so that
    staging blocks and accumulators are reused many times; bit-equal to torch's separate operations, and with the GELU to the
    same tiles stored from registers."""
    xq, wq, sr, sc, b, want = _exact_gemm_operands(cuda_dev, M, N, K, dtype)
    gelu = {}
    for tma in (1, 0):
        for ctas in (0, 4):
            gemm_options(gemm_pair=2, gemm_block_n=256, gemm_epi_warps=16, gemm_tma_store=tma, gemm_max_ctas=ctas)
            assert torch.equal(int8_exec.int8_gemm_fused(xq, sr, wq, sc, b, dtype), want), (tma, ctas)
            if N % 32 == 0:
                gelu[tma, ctas] = ops._gemm_impl(xq, sr, wq, sc, b, None, None, dtype, epilogue=ops.EPI_GELU_TANH)
    assert all(torch.equal(v, next(iter(gelu.values()))) for v in gelu.values())
    ops.check_device_status(cuda_dev)


@pytest.mark.parametrize("M,N,K", [(4096, 640, 2560), (4096, 640, 5120), (5000, 640, 640), (9600, 320, 320), (1024, 2376, 1808),
                                   (700, 3072, 1024), (2048, 264, 96)])
def test_gemm_kernel_choice_by_size(cuda_dev, gemm_options, M, N, K):
    """On both sides of the lines between the CTA-pair and the single-CTA kernel: the automatic choice, each kernel forced, and
    the single-CTA kernel with few CTAs give the same bits, one and two weight tiers, an output with and without room for the
    staged store; with the rank-32 term they agree to its rounding."""
    dtype = torch.bfloat16
    xq, wq, sr, sc, b, want = _exact_gemm_operands(cuda_dev, M, N, K, dtype)
    mh = M // 2 + 3
    tiers = torch.cat([want[:mh], (((xq[mh:].double() @ -wq.double().t()).float() * (sr[mh:, None] * (sc * 2)[None, :]))
                                   + b[None, :]).to(dtype)])
    g = torch.Generator(device="cuda").manual_seed(N)
    t = torch.randn(M, 32, generator=g, device=cuda_dev).to(dtype)
    lb = (torch.randn(32, N, generator=g, device=cuda_dev) * 0.1).to(dtype)
    lr = []
    for opt in ({}, {"gemm_pair": 2}, {"gemm_pair": 0}, {"gemm_pair": 0, "gemm_max_ctas": 3}, {"gemm_max_ctas": 6}):
        gemm_options(**opt)
        assert torch.equal(int8_exec.int8_gemm_fused(xq, sr, wq, sc, b, dtype), want), opt
        odd = torch.zeros(M, N + 2, dtype=dtype, device=cuda_dev)[:, :N]            # rows of no 16-byte pitch
        assert torch.equal(ops._gemm_impl(xq, sr, wq, sc, b, None, None, dtype, out=odd), want), opt
        assert torch.equal(int8_exec.int8_gemm_grouped(xq, sr, wq, sc, -wq, sc * 2, b, None, None, mh, dtype), tiers), opt
        lr.append(int8_exec.int8_gemm_lr(xq, sr, wq, sc, b, t, lb, dtype))
    ref = want.double() + t.double() @ lb.double()
    for y in lr:
        # one rounding of the output and one of the intermediate `want`, each at most 2^-9 of its operand
        assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * (want.double().abs() + ref.abs()) + 1e-6 * (t.double().abs() @ lb.double().abs())).all())
    ops.check_device_status(cuda_dev)


@pytest.mark.parametrize("pair", [0, 2])
def test_gemm_accumulators_beyond_24_bits_round_like_the_restatement(cuda_dev, pair):
    """Same-sign codes and K = 8192 give accumulators of 2^24 .. 2^27 with arbitrary low bits: the int32 -> fp32
    conversion of the epilogue has to round them to nearest-even exactly like the fp32 restatement.  Scales of 1 and
    no bias, fp16 and bf16 outputs of power-of-two-scaled sums expose the conversion's rounding at output ties."""
    g = torch.Generator().manual_seed(5)
    M, N, K = 512, 512, 8192
    xq = torch.randint(0, 128, (M, K), generator=g, dtype=torch.int8)
    wq = torch.randint(0, 128, (N, K), generator=g, dtype=torch.int8)
    wq[::2] = -wq[::2]
    acc = oracle.int_mm(xq, wq)
    assert int(acc.abs().max()) > 2 ** 24
    d = cuda_dev
    _lib.set_option("gemm_pair", pair)
    try:
        for dtype, sr_v in ((torch.bfloat16, 1.0), (torch.float16, 2.0 ** -12), (torch.bfloat16, 2.0 ** -7)):
            sr = torch.full((M,), sr_v); sc = torch.ones(N)
            want = oracle.epilogue(acc, sr, sc, None, None, None, dtype)
            got = int8_exec.int8_gemm_fused(xq.to(d), sr.to(d), wq.to(d), sc.to(d), None, dtype)
            assert torch.equal(got.cpu(), want), (pair, dtype)
    finally:
        _lib.set_option("gemm_pair", 1)


def test_gemm_cfg0_layer(cuda_dev):
    """M=4608, K=N=3072, rank-32 branch and bias, through Int8Linear.forward."""
    L = oracle.make_layer(0, 4608, 3072, 3072)
    lin = nn.Linear(3072, 3072, bias=True).to(torch.bfloat16)
    with torch.no_grad():
        lin.weight.copy_(L["w"]); lin.bias.copy_(L["bias"].to(torch.bfloat16))
    q = int8_exec.Int8Linear(lin, device=cuda_dev, lowrank=(L["lr_A"], L["lr_B"]))
    wq, ws = oracle.quant_weight(L["w"], where="cuda")
    assert torch.equal(q.weight_int8.cpu(), wq) and torch.equal(q.w_scale.cpu(), ws)
    x = L["x"].to(cuda_dev)
    y = q(x)
    assert y.dtype == torch.bfloat16 and y.shape == (4608, 3072)
    # integer stages bit-exact
    xq, sx = int8_exec.quant_rows(x)
    xqo, sxo = oracle.quant_rows(L["x"])
    assert torch.equal(xq.cpu(), xqo) and torch.equal(sx.cpu(), sxo)
    t_gpu = q._down(x)
    _, acc = ops.int8_gemm_debug(xq, sx, q.weight_int8, q.w_scale, q.bias, t_gpu, q.lr_B, torch.bfloat16)
    acc_ref = oracle.int_mm(xqo, wq)
    assert torch.equal(acc.cpu(), acc_ref)
    # output against the exact dequantised math and against the restated forward
    bias32 = lin.bias.detach().float()
    # the down-projection t = x @ lr_A (reference :390) accumulates in fp32 in another order than the CPU; its rounding
    # to bf16 may differ by one ulp, so the GEMM is judged on the t it was given and t on its own
    t_ref = (L["x"].float() @ L["lr_A"].float()).to(torch.bfloat16)
    assert bool(((t_gpu.cpu().float() - t_ref.float()).abs() <= t_ref.float().abs() * 2.0 ** -7 + 1e-3).all())
    ref64 = oracle.exact_dequant_f64(acc_ref, sxo, ws, bias32, t_gpu.cpu(), L["lr_B"])
    assert max_rel_err(y.cpu(), ref64) <= TOL
    y_or = oracle.int8_linear_forward(L["x"], wq, ws, bias32, L["lr_A"], L["lr_B"])
    rel_l2 = ((y.cpu().float() - y_or.float()).norm() / y_or.float().norm()).item()
    assert rel_l2 < 1e-3, rel_l2
    # 3-D input gives the same rows (reference self-test vi)
    y3 = q(x[:2048].reshape(8, 256, 3072))
    assert torch.equal(y3.reshape(2048, -1), q(x[:2048]))


def test_gemm_grouped_two_tiers(cuda_dev):
    g = torch.Generator().manual_seed(21)
    M, N, K, m_hi = 1000, 768, 512, 389
    xq = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8)
    w8 = torch.randint(-127, 128, (N, K), generator=g, dtype=torch.int8)
    s8 = torch.rand(N, generator=g) * 0.002 + 1e-4
    w4, s4 = oracle.nested4_from_int8(w8, s8)
    sr = torch.rand(M, generator=g) * 0.05 + 0.001
    b = torch.randn(N, generator=g) * 0.01
    t = torch.randn(M, 32, generator=g).to(torch.bfloat16)
    lb = (torch.randn(32, N, generator=g) * 0.02).to(torch.bfloat16)
    d = cuda_dev
    for mh in (m_hi, 0, M, 128):
        y = int8_exec.int8_gemm_grouped(xq.to(d), sr.to(d), w8.to(d), s8.to(d), w4.to(d), s4.to(d), b.to(d),
                                        t.to(d), lb.to(d), mh, torch.bfloat16).cpu()
        ref = torch.empty(M, N, dtype=torch.float64)
        ref[:mh] = oracle.exact_dequant_f64(oracle.int_mm(xq[:mh], w8), sr[:mh], s8, b, t[:mh], lb) if mh else ref[:mh]
        if mh < M:
            ref[mh:] = oracle.exact_dequant_f64(oracle.int_mm(xq[mh:], w4), sr[mh:], s4, b, t[mh:], lb)
        assert max_rel_err(y, ref) <= TOL, mh
        # the same call on the CTA-pair kernel (K-major low-rank factor given, kernel forced on): tiles of 256 rows
        # per tier, split rows not aligned to anything
        _lib.set_option("gemm_pair", 2)
        try:
            y2 = int8_exec.int8_gemm_grouped(xq.to(d), sr.to(d), w8.to(d), s8.to(d), w4.to(d), s4.to(d), b.to(d),
                                             t.to(d), lb.to(d), mh, torch.bfloat16, lb.t().contiguous().to(d)).cpu()
        finally:
            _lib.set_option("gemm_pair", 1)
        assert max_rel_err(y2, ref) <= TOL, mh


def test_shared_input_group(cuda_dev, monkeypatch):
    """Sibling layers on one input: one quantisation and one down-projection for the group, outputs identical to
    the same layers run alone on the same codes and the same slice of the shared down-projection."""
    g = torch.Generator().manual_seed(33)
    K, Ns, M = 512, (256, 512, 1024, 264), 700
    layers = []
    for i, N in enumerate(Ns):
        lin = nn.Linear(K, N, bias=(i != 1)).to(torch.bfloat16)
        with torch.no_grad():
            lin.weight.copy_(torch.randn(N, K, generator=g) * 0.02)
        lr = None if i == 2 else ((torch.randn(K, 32, generator=g) * 0.02).to(torch.bfloat16),
                                  (torch.randn(32, N, generator=g) * 0.02).to(torch.bfloat16))
        layers.append(int8_exec.Int8Linear(lin, device=cuda_dev, lowrank=lr))
    x = (torch.randn(2, M // 2, K, generator=g)).to(torch.bfloat16).to(cuda_dev)
    alone = [m(x) for m in layers]
    grp = int8_exec.share_input_quantisation(layers)
    calls = {"n": 0}
    real = ops._quant_rows_impl

    def counting(x2):
        calls["n"] += 1
        return real(x2)
    monkeypatch.setattr(ops, "_quant_rows_impl", counting)
    together = [m(x) for m in layers]
    assert calls["n"] == 1
    x2 = x.reshape(-1, K)
    xq, sx = real(x2)
    _xq, _sx, T = grp.prepare(x2)                      # the group's own down-projection of width 32 x members
    assert T.shape == (M, 32 * sum(m.lr_A is not None for m in layers))
    t_wide = (x2.float() @ torch.cat([m.lr_A for m in layers if m.lr_A is not None], dim=1).float()).to(torch.bfloat16)
    assert bool(((T.float() - t_wide.float()).abs() <= t_wide.float().abs() * 2.0 ** -7 + 1e-3).all())
    off = 0
    for m, ya, yt in zip(layers, alone, together):
        assert yt.shape == ya.shape == (2, M // 2, m.out_features)
        if m.lr_A is None:
            assert torch.equal(yt, ya)
            continue
        exp = int8_exec.int8_gemm_lr(xq, sx, m.weight_int8, m.w_scale, m.bias, T[:, off:off + 32], m.lr_B, torch.bfloat16)
        off += 32
        assert torch.equal(yt.reshape(M, -1), exp)
        assert max_rel_err(yt.float().cpu(), ya.double().cpu()) <= TOL      # down-projection may round differently
    # a modified input (same storage) is quantised again; so is a new tensor
    x.mul_(0.5)
    _ = layers[0](x)
    assert calls["n"] == 2
    _ = layers[1](x)
    assert calls["n"] == 2
    _ = layers[1](x.clone())
    assert calls["n"] == 3
    grp.clear()


@pytest.fixture
def epi_warps(request):
    """Epilogue warps of the CTA-pair kernel: the epilogue variants take that kernel at every size, sixteen warps at the sizes of
    these tests and eight in the large launches they stand for."""
    _lib.set_option("gemm_epi_warps", request.param)
    yield request.param
    _lib.set_option("gemm_epi_warps", 0)


def _toy_layer(cuda_dev, g, K, N, lowrank=True, bias=True, dtype=torch.bfloat16):
    lin = nn.Linear(K, N, bias=bias).to(dtype)
    with torch.no_grad():
        lin.weight.copy_(torch.randn(N, K, generator=g) * 0.05)
        if bias:
            lin.bias.copy_(torch.randn(N, generator=g) * 0.1)
    lr = ((torch.randn(K, 32, generator=g) * 0.05).to(dtype), (torch.randn(32, N, generator=g) * 0.05).to(dtype)) if lowrank else None
    return int8_exec.Int8Linear(lin, device=cuda_dev, lowrank=lr)


@pytest.mark.parametrize("epi_warps", [8, 16], indirect=True)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,lowrank", [(768, True), (512, False), (264, True)])
def test_epilogue_variants(cuda_dev, dtype, N, lowrank, epi_warps):
    """GELU(tanh) and accumulate-into-output in the GEMM epilogue against the separate torch kernels on the layer's own
    output: the sum bit for bit; the activation within two units in the last place of the output type (hardware tanh).
    N = 264 is a shape the fused variants do not take: same results through the unfused sequence."""
    g = torch.Generator().manual_seed(N + (1 if lowrank else 0))
    K, M = 512, 700
    layer = _toy_layer(cuda_dev, g, K, N, lowrank=lowrank, dtype=dtype)
    x = (torch.randn(M, K, generator=g) * 1.5).to(dtype).to(cuda_dev)
    y = layer(x)
    ref_act = F.gelu(y, approximate="tanh")
    got_act = layer.forward_ex(x, ops.EPI_GELU_TANH)
    ulp = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    err = (got_act.float() - ref_act.float()).abs()
    assert bool((err <= 2 * ulp * ref_act.float().abs() + 2e-3).all()), err.max().item()
    base = (torch.randn(M, N, generator=g)).to(dtype).to(cuda_dev)
    ref_sum = base + y
    out = base.clone()
    r = layer.forward_ex(x, ops.EPI_ACCUMULATE, out=out)
    assert r is out and torch.equal(out, ref_sum)
    both = base.clone()
    layer.forward_ex(x, ops.EPI_ACCUMULATE | ops.EPI_GELU_TANH, out=both)
    err = (both.float() - (base + ref_act).float()).abs()
    assert bool((err <= 4 * ulp * (base + ref_act).float().abs() + 4e-3).all()), err.max().item()


@pytest.mark.parametrize("epi_warps", [8, 16], indirect=True)
@pytest.mark.parametrize("M,K,N,lowrank,copies", [(700, 512, 768, True, 3), (1000, 256, 512, False, 7), (513, 3072, 1024, True, 1),
                                                  (300, 512, 264, True, 2)])
def test_gemm_stores_to_every_destination(cuda_dev, M, K, N, lowrank, copies, epi_warps):
    """`forward_into` (pq_int8_gemm_bcast): the epilogue writes each output tile to several buffers -- on several GPUs
    these are the peers' output buffers, here slices of larger local ones.  Every destination must equal the plain
    forward bit for bit and rows outside the slice must stay untouched.  N = 264 is a shape the kernel path does not
    take: same results through the copy path."""
    g = torch.Generator().manual_seed(M + copies)
    layer = _toy_layer(cuda_dev, g, K, N, lowrank=lowrank)
    x = (torch.randn(M, K, generator=g) * 1.5).to(torch.bfloat16).to(cuda_dev)
    ref = layer(x)
    pad = 40
    bufs = [torch.full((M + 2 * pad, N), 7.0, dtype=torch.bfloat16, device=cuda_dev) for _ in range(copies + 1)]
    views = [b[pad: pad + M] for b in bufs]
    r = layer.forward_into(x, views[0], views[1:])
    torch.cuda.synchronize()
    ops.check_device_status(cuda_dev)
    assert r.data_ptr() == views[0].data_ptr()
    for b, v in zip(bufs, views):
        assert torch.equal(v, ref)
        assert bool((b[:pad] == 7.0).all()) and bool((b[pad + M:] == 7.0).all())


def test_peer_store_gather_on_one_rank(cuda_dev):
    """`parallel.PeerStoreGather` without a process group: one rank owns all rows, the result is the layer's output."""
    from pyraquant_b200 import parallel
    g = torch.Generator().manual_seed(11)
    M, K, N = 900, 512, 768
    layer = _toy_layer(cuda_dev, g, K, N, lowrank=True)
    x = (torch.randn(M, K, generator=g) * 1.5).to(torch.bfloat16).to(cuda_dev)
    for chunks in (1, 3):
        og = parallel.PeerStoreGather(M, N, torch.bfloat16, cuda_dev, chunks=chunks)
        y = og.run(layer, x)
        assert y.shape == (M, N) and torch.equal(y, layer(x))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,K", [(1, 300, 3072), (2, 129, 640), (1, 70, 15360), (3, 50, 200), (1, 1, 1024)])
def test_adaln_quant_rows(cuda_dev, dtype, B, T, K):
    """LayerNorm + adaLN modulation + per-token quantisation in one kernel (flux/transformer_flux.py:236-239).  The
    quantisation of the modulated activations is exact; the modulated activations themselves equal the reference
    sequence (CPU restatement, and torch's own kernels on the GPU) except where the fp32 row statistics, summed in a
    different order, move a normalised value across a rounding boundary: a few elements in ten thousand, one unit in
    the last place of the products involved."""
    g = torch.Generator().manual_seed(B * 1000 + T + K)
    h = torch.randn(B, T, K, generator=g) * 2 + 0.3
    h[..., 5] *= 30.0
    h = h.to(dtype)
    scale = (torch.randn(B, K, generator=g) * 0.3).to(dtype)
    shift = (torch.randn(B, K, generator=g) * 0.2).to(dtype)
    hd, sc, sh = h.to(cuda_dev), scale.to(cuda_dev), shift.to(cuda_dev)
    q, s, z = ops.adaln_quant_rows(hd.reshape(-1, K), sc, sh, 1e-6, T)
    ops.check_device_status(cuda_dev)
    qo, so = oracle.quant_rows(z.cpu())
    assert torch.equal(q.cpu(), qo) and torch.equal(s.cpu(), so)
    q2, s2, none = ops.adaln_quant_rows(hd.reshape(-1, K), sc, sh, 1e-6, T, want_modulated=False)
    assert none is None and torch.equal(q2, q) and torch.equal(s2, s)
    ulp = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    refs = [oracle.adaln_modulate(h, scale, shift, 1e-6).reshape(-1, K),
            (F.layer_norm(hd, (K,), eps=1e-6) * (1 + sc[:, None]) + sh[:, None]).reshape(-1, K).cpu()]
    for zo in refs:
        diff = (z.cpu().float() - zo.float()).abs()
        bound = 4 * ulp * (zo.float().abs() + shift.float().abs().repeat_interleave(T, 0)) + 1e-6
        assert bool((diff <= bound).all()), (diff - bound).max().item()
        assert (z.cpu() != zo).float().mean().item() <= 2e-3


def test_forward_adaln(cuda_dev):
    """`Int8Linear.forward_adaln` against the separate sequence: torch's LayerNorm and modulation, then the layer."""
    g = torch.Generator().manual_seed(21)
    B, T, K, N = 2, 333, 1024, 768
    layer = _toy_layer(cuda_dev, g, K, N, lowrank=True)
    plain = _toy_layer(cuda_dev, g, K, N, lowrank=False)
    h = (torch.randn(B, T, K, generator=g) * 1.5).to(torch.bfloat16).to(cuda_dev)
    scale = (torch.randn(B, K, generator=g) * 0.3).to(torch.bfloat16).to(cuda_dev)
    shift = (torch.randn(B, K, generator=g) * 0.2).to(torch.bfloat16).to(cuda_dev)
    z_ref = F.layer_norm(h, (K,), eps=1e-6) * (1 + scale[:, None]) + shift[:, None]
    for m in (layer, plain):
        y, z = m.forward_adaln(h, scale, shift, return_modulated=True)
        assert y.shape == (B, T, N) and z.shape == h.shape
        assert (z != z_ref).float().mean().item() <= 2e-3
        assert torch.equal(y, m(z))                                  # the layer on the kernel's own modulated rows
        y_ref = m(z_ref)
        rel = ((y.float() - y_ref.float()).norm() / y_ref.float().norm()).item()
        assert rel < 2e-3, rel
        assert torch.equal(m.forward_adaln(h, scale, shift), y)
    # 2-D input with one modulation vector
    y2 = layer.forward_adaln(h[0], scale[0], shift[0])
    assert torch.equal(y2, layer.forward_adaln(h[:1], scale[:1], shift[:1])[0])


@pytest.mark.parametrize("epi_warps", [8, 16], indirect=True)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("K0,K1,lowrank", [(128, 160, True), (3072, 1024, True), (64, 16, False), (96, 160, True), (15360, 1024, False)])
def test_forward_on_two_sources(cuda_dev, dtype, K0, K1, lowrank, epi_warps):
    """`forward_cat(x0, x1)` == the layer on `torch.cat([x0, x1], -1)` (flux/transformer_flux.py:143-145), bit for bit:
    quantisation and down-projection read the two tensors in place.  K0 = 96 (seam off the 64-element grid) and
    K0 + K1 = 16384 (beyond the register-resident rows) take the concatenating route; row-strided views are consumed as
    they are.  Also through the gate-and-residual epilogue."""
    g = torch.Generator().manual_seed(K0 + K1)
    N, B, T = 256, 2, 150
    layer = _toy_layer(cuda_dev, g, K0 + K1, N, lowrank=lowrank, dtype=dtype)
    wide = (torch.randn(B, T, K0 + 40, generator=g) * 1.5).to(dtype).to(cuda_dev)
    x0 = wide[..., :K0]                                       # a view with a row stride of K0 + 40
    x1 = (torch.randn(B, T, K1, generator=g) * 0.7).to(dtype).to(cuda_dev)
    x1[..., 3] *= 25.0
    want = layer(torch.cat([x0, x1], dim=-1))
    got = layer.forward_cat(x0, x1)
    assert got.shape == want.shape and torch.equal(got, want)
    gate = (torch.randn(B, N, generator=g) * 0.5).to(dtype).to(cuda_dev)
    residual = torch.randn(B, T, N, generator=g).to(dtype).to(cuda_dev)
    ref = residual + gate.unsqueeze(1) * want
    res = residual.clone()
    layer.forward_gated_residual(x0, gate, res, x_more=x1)
    assert torch.equal(res, ref)
    ops.check_device_status(cuda_dev)


def test_shared_group_primed_by_adaln(cuda_dev, monkeypatch):
    """`SharedInputGroup.prime_adaln`: one pass produces the modulated activations and the members' shared codes; the
    members called on the result skip their own quantisation and give what they give ungrouped on the same tensor."""
    g = torch.Generator().manual_seed(41)
    B, T, K = 2, 200, 512
    layers = [_toy_layer(cuda_dev, g, K, n, lowrank=lr) for n, lr in ((768, True), (512, True), (256, False))]
    h = (torch.randn(B, T, K, generator=g) * 1.5).to(torch.bfloat16).to(cuda_dev)
    scale = (torch.randn(B, K, generator=g) * 0.3).to(torch.bfloat16).to(cuda_dev)
    shift = (torch.randn(B, K, generator=g) * 0.2).to(torch.bfloat16).to(cuda_dev)
    z_alone = ops.adaln_quant_rows(h.reshape(-1, K), scale, shift, 1e-6, T)[2].reshape(h.shape)
    want = [m(z_alone) for m in layers]
    grp = int8_exec.share_input_quantisation(layers)
    z = grp.prime_adaln(h, scale, shift)
    assert torch.equal(z, z_alone)
    calls = []
    real = ops._quant_rows_impl
    monkeypatch.setattr(ops, "_quant_rows_impl", lambda x2: (calls.append(1), real(x2))[1])
    got = [m(z) for m in layers]
    assert not calls, "members quantised again although the group was primed"
    for a, b, m in zip(got, want, layers):
        if m.lr_A is None:
            assert torch.equal(a, b)
        else:                                            # the shared down-projection is 64 columns wide: other fp32 summation order
            assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 2e-3


@pytest.mark.parametrize("epi_warps", [8, 16], indirect=True)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lowrank", [True, False])
def test_gated_residual_epilogue(cuda_dev, dtype, lowrank, epi_warps):
    """`residual + gate.unsqueeze(1) * Linear(x)` (flux/transformer_flux.py:145-149) in the GEMM epilogue: bit-identical to
    the layer followed by torch's multiply and add, two samples with their own gate vectors, fp16 sums clipped as the
    block clips them."""
    g = torch.Generator().manual_seed(31)
    B, T, K, N = 2, 333, 512, 768
    layer = _toy_layer(cuda_dev, g, K, N, lowrank=lowrank, dtype=dtype)
    x = (torch.randn(B, T, K, generator=g) * 1.5).to(dtype).to(cuda_dev)
    gate = (torch.randn(B, N, generator=g) * 0.7).to(dtype).to(cuda_dev)
    residual = (torch.randn(B, T, N, generator=g) * 3).to(dtype).to(cuda_dev)
    if dtype == torch.float16:
        residual[0, 0, :8] = 65000.0; residual[1, 5, :8] = -65000.0        # sums that leave the fp16 range
        gate[:, :8] = gate[:, :8].abs() + 40.0
    y = layer(x)
    want = residual + gate.unsqueeze(1) * y
    if dtype == torch.float16:
        want = want.clip(-65504, 65504)
    res = residual.clone()
    out = layer.forward_gated_residual(x, gate, res)
    assert out is res and torch.equal(res, want)
    # 2-D input, one gate vector
    res2 = residual[1].clone()
    layer.forward_gated_residual(x[1], gate[1], res2)
    assert torch.equal(res2, want[1])
    ops.check_device_status(cuda_dev)


def test_split_input_linear(cuda_dev):
    """y = L0(x[..., :in0]) + L1(x[..., in0:]) with the sum in the second GEMM's epilogue: identical to the two layers
    and a torch add (pyraquant/external_quant.py:191-192), 3-D input, strided halves."""
    g = torch.Generator().manual_seed(5)
    in0, in1, N = 256, 768, 512
    l0 = _toy_layer(cuda_dev, g, in0, N, lowrank=True, bias=False)
    l1 = _toy_layer(cuda_dev, g, in1, N, lowrank=True, bias=True)
    x = torch.randn(3, 333, in0 + in1, generator=g).to(torch.bfloat16).to(cuda_dev)
    ref = l0(x[..., :in0]) + l1(x[..., in0:])
    m = int8_exec.SplitInInt8Linear(l0, l1)
    y = m(x)
    assert y.shape == ref.shape and torch.equal(y, ref)


def test_forward_is_cuda_graph_capturable(cuda_dev):
    """After one warm-up call (library load, kernel attributes, tensor-map cache) a chain of Int8Linear forwards is
    captured into a CUDA graph and replayed on new input values: same bits as the eager calls."""
    g = torch.Generator().manual_seed(9)
    l0 = _toy_layer(cuda_dev, g, 512, 1024, lowrank=True)
    l1 = _toy_layer(cuda_dev, g, 1024, 512, lowrank=False)
    x = torch.randn(300, 512, generator=g).to(torch.bfloat16).to(cuda_dev)

    def chain():
        return l1(l0(x))
    chain(); chain()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y_static = chain()
    for seed in (1, 2):
        x.copy_(torch.randn(300, 512, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y_static, chain())
    ops.check_device_status(cuda_dev)


def test_packed_low_tier(cuda_dev):
    """Four-bit storage of the low tier: pack -> device expansion returns the codes bit for bit (every nibble value
    at every position of a byte), and the routed Linear built with packed storage gives the same output as the one
    that keeps int8 codes."""
    g = torch.Generator().manual_seed(12)
    codes = torch.randint(-8, 8, (37, 96), generator=g, dtype=torch.int8)
    codes[0, :16] = torch.arange(-8, 8, dtype=torch.int8)
    codes[1, :32] = torch.arange(-8, 8, dtype=torch.int8).repeat_interleave(2)
    packed = ops.pack_int4(codes)
    assert packed.shape == (37, 48) and packed.dtype == torch.uint8
    assert torch.equal(ops.unpack_int4(packed.to(cuda_dev)).cpu(), codes)
    K, N, M = 512, 768, 600
    lin = nn.Linear(K, N, bias=True).to(torch.bfloat16)
    A = (torch.randn(K, 32, generator=g) * 0.02).to(torch.bfloat16)
    B = (torch.randn(32, N, generator=g) * 0.02).to(torch.bfloat16)
    plain = int8_exec.Int8LinearRouted(lin, device=cuda_dev, lowrank=(A, B))
    small = int8_exec.Int8LinearRouted(lin, device=cuda_dev, lowrank=(A, B), pack_lo=True)
    assert small.weight_lo_packed.numel() * 2 == plain.weight_lo.numel() and not hasattr(small, "weight_lo")
    assert torch.equal(ops.unpack_int4(small.weight_lo_packed), plain.weight_lo)
    x = rand_act(M, K, torch.bfloat16, 13).to(cuda_dev)
    for m_hi in (0, 250, M):
        assert torch.equal(small.forward_rows(x, m_hi), plain.forward_rows(x, m_hi))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,R", [(1, 64, 32), (63, 128, 32), (64, 200, 32), (129, 3072, 32), (1000, 1288, 32),
                                   (4608, 3072, 32), (65, 200, 64), (1000, 1288, 96), (129, 3072, 128),
                                   (9500, 3072, 128), (9500, 512, 64)])
def test_lowrank_down_projection(cuda_dev, M, K, R, dtype):
    """t = x @ A on the streaming tensor-core kernel against the fp64 product: within one unit in the last place of
    the output type (fp32 accumulation order differs from any reference), identical to torch's own matmul almost
    everywhere; row tails, K tails (K % 64 != 0), strided rows, one to four rank-32 factors side by side."""
    g = torch.Generator().manual_seed(M + K + R)
    xp = torch.randn(M, K + 8, generator=g).to(dtype)
    x = xp[:, :K]
    A = (torch.randn(K, R, generator=g) * 0.05).to(dtype)
    xd, Ad = xp.to(cuda_dev)[:, :K], A.to(cuda_dev)                   # row stride K + 8 on the device too
    assert xd.stride(0) == K + 8 or M == 1
    t = ops.lowrank_down(xd, Ad.t().contiguous()).cpu()
    ref = x.double() @ A.double()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    err = (t.double() - ref).abs()
    mag = x.double().abs() @ A.double().abs()                        # bound of the fp32 accumulation error
    assert bool((err <= ulp * ref.abs() * 1.01 + 1e-6 * mag).all()), err.max().item()
    t_torch = (xd @ Ad).cpu()
    assert (t != t_torch).float().mean().item() < 0.02
    ops.check_device_status(cuda_dev)


def test_shared_input_group_uses_native_down_projection_for_many_rows(cuda_dev, monkeypatch):
    """A group of layers on one input takes ONE native down-projection of width 32 x members, and
    every member's output equals the ungrouped layer's wherever the two down-projections agree (they differ in fp32
    summation order only)."""
    from pyraquant_b200.int8_exec import share_input_quantisation
    g = torch.Generator().manual_seed(11)
    M, K = 32768 + 37, 256
    grouped = [_toy_layer(cuda_dev, g, K, n, lowrank=True) for n in (256, 512, 256)]
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).to(cuda_dev)
    alone = [m(x) for m in grouped]                                  # before grouping: one kernel call each
    t_alone = [m._down(x) for m in grouped]
    calls = []
    real = ops.lowrank_down

    def counting(x2, a_t):
        calls.append(tuple(a_t.shape))
        return real(x2, a_t)

    monkeypatch.setattr(ops, "lowrank_down", counting)
    grp = share_input_quantisation(grouped)
    outs = [m(x) for m in grouped]
    assert calls == [(96, K)], calls
    _, _, T = grp.prepare(x)
    for i, m in enumerate(grouped):
        same_t = (grp.t_of(m, T) == t_alone[i]).all(dim=1)
        assert same_t.float().mean().item() > 0.9
        assert torch.equal(outs[i][same_t], alone[i][same_t])
        assert (outs[i].float() - alone[i].float()).abs().max().item() <= 0.02 * alone[i].float().abs().max().item()
    ops.check_device_status(cuda_dev)


def test_int8linear_uses_native_down_projection_for_many_rows(cuda_dev, monkeypatch):
    """Int8Linear.forward takes the library's own down-projection kernel at small and large row counts: the output
    matches the exact dequantised math built on that kernel's t, and the kernel really is the one called."""
    g = torch.Generator().manual_seed(3)
    M, K, N = 32768 + 100, 256, 256
    layer = _toy_layer(cuda_dev, g, K, N, lowrank=True)
    x = (torch.randn(M, K, generator=g)).to(torch.bfloat16)
    calls = {"n": 0}
    real = ops.lowrank_down

    def counting(x2, a_t):
        calls["n"] += 1
        return real(x2, a_t)
    monkeypatch.setattr(ops, "lowrank_down", counting)
    xd = x.to(cuda_dev)
    y = layer(xd).cpu()
    assert calls["n"] == 1
    t = real(xd, layer._lr_At()).cpu()
    xq, sx = oracle.quant_rows(x)
    ref = oracle.exact_dequant_f64(oracle.int_mm(xq, layer.weight_int8.cpu()), sx, layer.w_scale.cpu(), layer.bias.cpu(),
                                   t, layer.lr_B.cpu())
    assert max_rel_err(y, ref) <= TOL


def test_dequant_epilogue_and_linear_2d(cuda_dev):
    L = oracle.make_layer(5, 300, 512, 256, lowrank=False)
    wq, ws = oracle.quant_weight(L["w"], where="cuda")
    xq, sx = oracle.quant_rows(L["x"])
    acc = oracle.int_mm(xq, wq)
    d = cuda_dev
    y = int8_exec.dequant_epilogue(acc.to(d), sx.to(d), ws.to(d), L["bias"].to(d), torch.bfloat16)
    assert torch.equal(y.cpu(), oracle.epilogue(acc, sx, ws, L["bias"], None, None, torch.bfloat16))
    for backend in (None, "triton", "cublas"):
        y2 = int8_exec.int8_linear_2d(L["x"].to(d), wq.to(d), ws.to(d), L["bias"].to(d), backend=backend)
        assert max_rel_err(y2.cpu(), oracle.exact_dequant_f64(acc, sx, ws, L["bias"], None, None)) <= TOL
    with pytest.raises(ValueError):
        int8_exec.int8_linear_2d(L["x"].to(d), wq.to(d), ws.to(d), None, backend="nope")


def test_reference_selftest_assertions(cuda_dev):
    """The reference's own numerical self-test (deploy/int8_exec.py:498-536) with its thresholds."""
    rep = int8_exec.selftest_and_bench(Ms=())["selftest"]
    assert rep["act_quant_mismatch_elems"] == 0 and rep["act_scale_max_rel_err"] == 0.0


# ------------------------------------------------------------------------------------------------ group-32 path
@pytest.mark.parametrize("M,K,N", [(128, 128, 128), (300, 640, 640), (257, 1280, 1280), (1000, 2560, 640),
                                   (77, 640, 5120), (512, 5120, 1280), (130, 256, 264)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gemm_g32_matches_oracle(cuda_dev, M, K, N, dtype):
    """SDXL W8A8 group-32 shapes (config 3) in miniature: integer grid from the oracle, GEMM on the GPU."""
    g = torch.Generator().manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g).to(dtype)
    w = torch.randn(N, K, generator=g) * 0.02
    b = torch.randn(N, generator=g) * 0.01
    xq, sa = oracle.quant_rows_g32(x)
    wq, sw = oracle.quant_weight_g32(w, where="cuda")
    d = cuda_dev
    for bias in (b, None):
        y = int8_exec.int8_gemm_g32(xq.to(d), sa.to(d), wq.to(d), sw.t().contiguous().to(d),
                                    None if bias is None else bias.to(d), dtype).cpu()
        want = oracle.gemm_g32(xq, sa, wq, sw, bias, dtype)
        assert torch.equal(y, want)                  # exact partial sums and the same fp32 operation order
        assert max_rel_err(y, oracle.gemm_g32_f64(xq, sa, wq, sw, bias)) <= TOL


def test_int8linear_g32_module(cuda_dev):
    g = torch.Generator().manual_seed(33)
    lin = nn.Linear(640, 1280, bias=True)
    with torch.no_grad():
        lin.weight.copy_(torch.randn(1280, 640, generator=g) * 0.02); lin.bias.copy_(torch.randn(1280, generator=g) * 0.01)
    x = torch.randn(3, 77, 640, generator=g).to(torch.float16)
    q = int8_exec.Int8LinearG32(lin.to(torch.float16), device=cuda_dev)
    wq, sw = oracle.quant_weight_g32(lin.weight.detach().float(), where="cuda")
    assert torch.equal(q.weight_int8.cpu(), wq) and torch.equal(q.w_scale.cpu(), sw)
    y = q(x.to(cuda_dev)).cpu()
    xq, sa = oracle.quant_rows_g32(x.reshape(-1, 640))
    want = oracle.gemm_g32(xq, sa, wq, sw, lin.bias.detach().float(), torch.float16).reshape(3, 77, 1280)
    assert torch.equal(y, want)
    assert set(q.state_dict()) == {"weight_int8", "w_scale", "bias"}


# ------------------------------------------------------------------------------------------------ full-size properties
def test_full_size_quant_and_gemm_properties(cuda_dev):
    """BASELINE config 2 row count (M = 65536 + 512) at K = 3072 -> N = 3072: sizes the CPU oracle cannot
    finish quickly, so parity is checked through exact size-independent identities:
      column checksum  sum_m acc[m,:] == (sum_m xq[m,:]) @ w^T        (int64, exact)
      row checksum     sum_n acc[m,:] == xq[m,:] @ (sum_n w[n,:])     (int64, exact)
    plus the per-row quantisation identities |x - q*s| <= s/2 and max|q| == 127."""
    d = cuda_dev
    M, K, N = 66048, 3072, 3072
    g = torch.Generator(device=d).manual_seed(2)
    x = torch.randn(M, K, generator=g, device=d, dtype=torch.float32)
    x[:, ::211] *= 20.0
    x = x.to(torch.bfloat16)
    q, s = int8_exec.quant_rows(x)
    xf = x.float()
    amax = xf.abs().amax(1).clamp_min(1e-8)
    s_ref = amax / torch.full_like(amax, 127.0)            # tensor / tensor: IEEE division on CUDA as well
    assert torch.equal(s, s_ref)
    assert int(q.abs().amax(1).min()) == 127
    assert bool(((xf - q.float() * s[:, None]).abs() <= s[:, None] * 0.5001).all())
    del xf
    w = torch.randint(-127, 128, (N, K), generator=g, device=d, dtype=torch.int8)
    sc = torch.rand(N, generator=g, device=d) * 1e-3 + 1e-4
    out, acc = ops.int8_gemm_debug(q, s, w, sc, None, None, None, torch.bfloat16)
    col = acc.sum(0, dtype=torch.int64).cpu()
    row = acc.sum(1, dtype=torch.int64).cpu()
    qs = q.sum(0, dtype=torch.int64).cpu()
    ws = w.sum(0, dtype=torch.int64).cpu()
    assert torch.equal(col, w.cpu().to(torch.int64) @ qs)
    row_ref = torch.empty(M, dtype=torch.int64)
    qc = q.cpu()
    for i in range(0, M, 8192):
        row_ref[i:i + 8192] = qc[i:i + 8192].to(torch.int64) @ ws
    assert torch.equal(row, row_ref)
    # output = rounding of acc * (s_row*s_col): recompute from the verified accumulators in chunks
    for i in range(0, M, 16384):
        ref = (acc[i:i + 16384].float() * (s[i:i + 16384, None] * sc[None, :])).to(torch.bfloat16)
        assert torch.equal(out[i:i + 16384], ref)


# ------------------------------------------------------------------------------------------------ gather / scatter
def test_scatter_matches_reference_fixture(cuda_dev, golden):
    g = golden("routing_gather_scatter.npz")
    boxes = [tuple(b) for b in g["boxes"].tolist()]
    bg = from_bf16_bits(g["background_bits"])
    for prefix, halo, fb, bx, key in (("", 2, 1.0, boxes, "n_buckets"), ("h3_", 3, 0.75, boxes[:4], "h3_n_buckets")):
        plan = routing.build_route_plan((24, 24), bx, halo, fusion_beta=fb)
        y = torch.cat([from_bf16_bits(g[f"{prefix}bucket{i}_out_bits"]).reshape(-1, bg.shape[-1])
                       for i in range(int(g[key]))])
        fused = routing.fuse_rows(bg.to(cuda_dev), y.to(cuda_dev), plan)
        assert torch.equal(fused.cpu(), from_bf16_bits(g[f"{prefix}fused_bits"]))
    hidden = from_bf16_bits(g["hidden_bits"]).reshape(24 * 24, -1)
    plan = routing.build_route_plan((24, 24), boxes, 2)
    got = routing.gather_rows(hidden.to(cuda_dev), plan)
    want = torch.cat([from_bf16_bits(g[f"bucket{i}_hidden_bits"]).reshape(-1, hidden.shape[1])
                      for i in range(int(g["n_buckets"]))])
    assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_routed_gather_scatter_vs_oracle(cuda_dev, dtype):
    """64x64 token canvas, 8x8 leaves of 8 tokens, Bernoulli(0.3) selection, halo 2, C = 256."""
    H = W = 64; C = 256
    g = torch.Generator().manual_seed(4)
    sel = (torch.rand(8, 8, generator=g) < 0.3).float().numpy()
    boxes = routing.leaf_run_boxes(sel, 16)                     # leaf = 16 latent = 8 tokens
    canvas = torch.randn(1, H, W, C, generator=g).to(dtype)
    bg = torch.randn(1, H, W, C, generator=g).to(dtype)
    plan = routing.build_route_plan((H, W), boxes, 2, dtype=dtype)
    buckets = oracle.gather_buckets(canvas, boxes, 2)
    want_rows = torch.cat([t.reshape(-1, C) for _hw, t, _g in buckets])
    d = cuda_dev
    rows = routing.gather_rows(canvas.reshape(H * W, C).to(d), plan)
    assert torch.equal(rows.cpu(), want_rows)
    q, s = routing.gather_quant_rows(canvas.reshape(H * W, C).to(d), plan)
    qo, so = oracle.quant_rows(want_rows)
    assert torch.equal(q.cpu(), qo) and torch.equal(s.cpu(), so)
    outs, ys = [], []
    for hw, t, geoms in buckets:
        o = (torch.randn(t.shape, generator=g) * 2).to(dtype)
        # signed zeros in the routed rows (and a background of both signs): 0 * bg + y keeps or drops the sign of a zero
        # exactly as the reference's arithmetic does
        o.view(-1)[torch.randperm(o.numel(), generator=g)[: o.numel() // 50]] = -0.0
        o.view(-1)[torch.randperm(o.numel(), generator=g)[: o.numel() // 50]] = 0.0
        outs.append(((hw, geoms), o)); ys.append(o.reshape(-1, C))
    want = oracle.fuse_buckets(bg, outs, 1.0)
    got = routing.fuse_rows(bg.to(d), torch.cat(ys).to(d), plan)
    assert torch.equal(got.cpu().view(torch.int16), want.view(torch.int16))       # bit patterns: -0 and +0 differ
    # untouched tokens are bit-identical to the background
    touched = torch.zeros(H * W, dtype=torch.bool); touched[torch.from_numpy(plan.tokens).long()] = True
    assert torch.equal(got.cpu().reshape(H * W, C)[~touched], bg.reshape(H * W, C)[~touched])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_scatter_contributor_lists_of_every_kind(cuda_dev, dtype):
    """`pq_scatter_rows` on hand-made contributor lists that the routing plans of the other tests do not produce: one
    full-weight contributor (copied), fractional weights, weights that are not values of the canvas type (fp32
    arithmetic instead of the packed one), two and five contributors, more than 32 (the list is then walked from global
    memory), out-of-range row numbers (skipped), an all-invalid list (weight sum 0), signed zeros.  Checked bit for bit
    against the reference's sequence of roundings evaluated in fp32 with explicit rounding after every step."""
    g = torch.Generator().manual_seed(77)
    C, M_act, rows = 264, 64, 40
    y = (torch.randn(M_act, C, generator=g) * 2).to(dtype)
    y[3, :20] = -0.0; y[5, 7] = 0.0
    canvas = torch.randn(rows, C, generator=g).to(dtype)
    canvas[2, :9] = -0.0
    q = lambda v: float(torch.tensor(v).to(dtype))                     # a weight representable in the canvas type
    lists = [
        [(3, 1.0)],                                                       # copy, with -0 in the row
        [(7, q(0.37))],                                                   # one fractional weight: background keeps a share
        [(8, 0.3)],                                                       # 0.3 is not a bf16 / fp16 value
        [(1, 1.0), (2, q(0.25))],                                         # sum > 1, two contributors
        [(9, q(0.5)), (10, q(0.5))],                                      # power-of-two divisor
        [(11, q(0.2)), (12, q(0.3)), (13, q(0.1)), (14, q(0.15)), (15, q(0.05))],
        [(i % M_act, q(0.02)) for i in range(40)],                        # more than 32 entries
        [(-1, 1.0), (5, 1.0)],                                            # an invalid row number in front of a valid one
        [(M_act + 3, q(0.5))],                                            # nothing valid: weight sum 0
        [(20, 1.0), (-5, q(0.5)), (21, q(0.125))],
    ]
    tokens = torch.tensor([0, 2, 5, 6, 9, 17, 18, 30, 31, 39], dtype=torch.int32)
    ptr, src, beta = [0], [], []
    for lst in lists:
        src += [r for r, _ in lst]; beta += [b for _, b in lst]; ptr.append(len(src))
    rnd = lambda t: t.to(dtype).float()
    want = canvas.clone()
    for tok, lst in zip(tokens.tolist(), lists):
        local = torch.zeros(C); bsum = torch.zeros(())
        for r, b in lst:
            if r < 0 or r >= M_act:
                continue
            bt = torch.tensor(b, dtype=torch.float32)
            local = rnd(local + rnd(bt * y[r].float()))
            bsum = rnd(bsum + bt)
        bm = bsum.clamp(0.0, 1.0)
        denom = rnd(bsum.clamp_min(1e-8))
        om = rnd(1.0 - bm)
        c = rnd(local / denom) if bsum > 0 else torch.zeros(C)
        want[tok] = (rnd(om * canvas[tok].float()) + rnd(bm * c)).to(dtype)
    got = canvas.clone().to(cuda_dev)
    ops._scatter_rows_impl(y.to(cuda_dev), tokens.to(cuda_dev), torch.tensor(ptr, dtype=torch.int32, device=cuda_dev),
                           torch.tensor(src, dtype=torch.int32, device=cuda_dev),
                           torch.tensor(beta, dtype=torch.float32, device=cuda_dev), got)
    torch.cuda.synchronize()
    assert torch.equal(got.cpu().view(torch.int16), want.view(torch.int16))


def test_routed_two_tier_linear(cuda_dev):
    """Config-4 shape in miniature: routed rows -> Linear with per-leaf hi/lo weights -> scatter."""
    H = W = 32; K = 256; N = 512
    g = torch.Generator().manual_seed(8)
    sel = (torch.rand(4, 4, generator=g) < 0.4).float().numpy(); sel[0, 0] = 1; sel[1, 0] = 1
    scores = torch.rand(4, 4, generator=g).numpy()
    hi = routing.inner_split_median(scores, sel, 1.0)
    tmap = routing.leaf_tier_to_token_map(hi, (H, W))
    plan = routing.build_route_plan((H, W), routing.leaf_run_boxes(sel, 16), 2, token_tier_hi=tmap)
    canvas = rand_act(H * W, K, torch.bfloat16, 31)
    lin = nn.Linear(K, N, bias=True).to(torch.bfloat16)
    A = (torch.randn(K, 32, generator=g) * 0.02).to(torch.bfloat16)
    B = (torch.randn(32, N, generator=g) * 0.02).to(torch.bfloat16)
    q = int8_exec.Int8LinearRouted(lin, device=cuda_dev, lowrank=(A, B))
    y = q.forward_gathered(canvas.to(cuda_dev), plan.to(cuda_dev)["row_idx"], plan.m_hi).cpu()
    rows = canvas[torch.from_numpy(plan.row_idx).long()]
    w8, s8 = oracle.quant_weight(lin.weight.detach(), where="cuda")
    w4, s4 = oracle.nested4_from_int8(w8, s8)
    xq, sx = oracle.quant_rows(rows)
    t = q._down(rows.to(cuda_dev)).cpu()                      # the module's own down-projection
    b32 = lin.bias.detach().float()
    mh = plan.m_hi
    ref = torch.cat([oracle.exact_dequant_f64(oracle.int_mm(xq[:mh], w8), sx[:mh], s8, b32, t[:mh], B),
                     oracle.exact_dequant_f64(oracle.int_mm(xq[mh:], w4), sx[mh:], s4, b32, t[mh:], B)])
    assert 0 < mh < plan.n_rows
    assert max_rel_err(y, ref) <= TOL
    y2 = q.forward_rows(rows.to(cuda_dev), mh).cpu()
    assert max_rel_err(y2, ref) <= TOL


@pytest.mark.parametrize("case", ["rank16", "fp16_factors"])
def test_routed_linear_keeps_a_lowrank_branch_it_cannot_fuse(cuda_dev, case):
    """A low-rank branch outside the fused epilogue's reach (rank 16; factors in another dtype than the activations)
    is added after the two-tier GEMM instead of being dropped."""
    H = W = 16; K = 128; N = 256
    g = torch.Generator().manual_seed(90)
    sel = np.zeros((2, 2), np.float32); sel[0, 0] = sel[1, 1] = 1
    tmap = routing.leaf_tier_to_token_map(np.array([[1, 0], [0, 0]], np.float32), (H, W))
    plan = routing.build_route_plan((H, W), routing.leaf_run_boxes(sel, 16), 2, token_tier_hi=tmap)
    canvas = rand_act(H * W, K, torch.bfloat16, 91)
    lin = nn.Linear(K, N, bias=True).to(torch.bfloat16)
    R, fdt = (16, torch.bfloat16) if case == "rank16" else (32, torch.float16)
    A = (torch.randn(K, R, generator=g) * 0.05).to(fdt)
    B = (torch.randn(R, N, generator=g) * 0.05).to(fdt)
    q = int8_exec.Int8LinearRouted(lin, device=cuda_dev, lowrank=(A, B))
    rows = canvas[torch.from_numpy(plan.row_idx).long()]
    w8, s8 = oracle.quant_weight(lin.weight.detach(), where="cuda")
    w4, s4 = oracle.nested4_from_int8(w8, s8)
    xq, sx = oracle.quant_rows(rows)
    t = (rows.to(fdt).float() @ A.float()).to(fdt)
    b32 = lin.bias.detach().float()
    mh = plan.m_hi
    assert 0 < mh < plan.n_rows
    # the unfused sequence rounds twice (the GEMM output, then the sum), like the reference's own unfused branch
    # (deploy/int8_exec.py:394-407): the bar is the exact sum of the ROUNDED GEMM output and the exact low-rank term
    y_gemm = torch.cat([oracle.epilogue(oracle.int_mm(xq[:mh], w8), sx[:mh], s8, b32, None, None, torch.bfloat16),
                        oracle.epilogue(oracle.int_mm(xq[mh:], w4), sx[mh:], s4, b32, None, None, torch.bfloat16)])
    branch = t.double() @ B.double()
    ref = y_gemm.double() + branch
    assert float(branch.abs().mean() / y_gemm.double().abs().mean()) > 0.05      # the branch matters in this case
    # every rounding on the way (the factors and t converted to the activation dtype, GEMM output, the library's
    # product, the sum) is at most half a unit in the last place of its operand: the result stays within 2^-7 of the
    # operands' magnitudes of the exact sum, element by element
    bound = 2.0 ** -7 * (y_gemm.double().abs() + t.double().abs() @ B.double().abs()) + 1e-30

    def close(y):
        d = (y.double() - ref).abs()
        return bool((d <= bound).all()) and float(d.norm() / ref.norm()) < 4e-3

    y = q.forward_gathered(canvas.to(cuda_dev), plan.to(cuda_dev)["row_idx"], mh).cpu()
    assert close(y)
    assert max_rel_err(y, y_gemm.double()) > 5 * TOL               # i.e. the branch was not dropped
    y2 = q.forward_rows(rows.to(cuda_dev), mh).cpu()
    assert close(y2)


def test_shared_input_group_under_inference_mode_and_after_inplace_writes(cuda_dev, monkeypatch):
    """Inference tensors keep no version counter: grouped layers then run ungrouped instead of failing.  The
    library's own in-place write (accumulate epilogue) bumps the version of its target, so a cached quantisation of
    that tensor is not reused afterwards."""
    g = torch.Generator().manual_seed(34)
    K = 256
    a, b = _toy_layer(cuda_dev, g, K, 256), _toy_layer(cuda_dev, g, K, 256)
    x = rand_act(300, K, torch.bfloat16, 35).to(cuda_dev)
    alone = [a(x), b(x)]
    int8_exec.share_input_quantisation([a, b])
    with torch.inference_mode():
        xi = x.clone()
        assert xi.is_inference()
        got = [a(xi), b(xi)]
    assert torch.equal(got[0], alone[0]) and torch.equal(got[1], alone[1])
    # accumulate into a tensor the group has cached, then feed it to the group again
    calls = {"n": 0}
    real = ops._quant_rows_impl

    def counting(x2):
        calls["n"] += 1
        return real(x2)
    monkeypatch.setattr(ops, "_quant_rows_impl", counting)
    h = x.clone()
    y0 = a(h)                                                       # caches the quantisation of h
    n0 = calls["n"]
    v0 = h._version
    c = _toy_layer(cuda_dev, g, K, K, lowrank=False)
    c.forward_ex(x, ops.EPI_ACCUMULATE, out=h)                      # h += c(x), written by the GEMM epilogue
    assert h._version > v0
    y1 = b(h)
    assert calls["n"] == n0 + 2 and not torch.equal(h, x)         # c quantised x, b quantised the updated h
    monkeypatch.setattr(ops, "_quant_rows_impl", real)
    b.__dict__.pop("_shared_input"); a.__dict__.pop("_shared_input")
    assert torch.equal(y1, b(h))                                    # the fresh codes, not the stale ones
    del y0


def test_lean_path_follows_converted_buffers(cuda_dev):
    """Replacing or converting the float buffers (w_scale, bias, lr_B) while the int8 weight stays in place must not
    leave the fast path with stale addresses."""
    g = torch.Generator().manual_seed(36)
    m = _toy_layer(cuda_dev, g, 256, 512)
    x = rand_act(200, 256, torch.bfloat16, 37).to(cuda_dev)
    y0 = m(x)
    with torch.no_grad():
        new_scale = (m.w_scale * 2.0).clone()
        new_B = (m.lr_B.float() * 0.5).to(torch.bfloat16)
    m.w_scale = new_scale
    m.lr_B = new_B
    y1 = m(x)
    xq, sx = int8_exec.quant_rows(x)
    want = int8_exec.int8_gemm_lr(xq, sx, m.weight_int8, new_scale, m.bias, m._down(x), new_B, torch.bfloat16)
    assert torch.equal(y1, want) and not torch.equal(y1, y0)
    m.lr_B.mul_(2.0)                                               # in place: the K-major copy must follow
    want2 = int8_exec.int8_gemm_lr(xq, sx, m.weight_int8, new_scale, m.bias, m._down(x), m.lr_B, torch.bfloat16)
    assert torch.equal(m(x), want2)


def test_bounded_wait_runs_out_and_is_reported(cuda_dev):
    """A device-side wait that nothing ends: the kernel gives up after its budget (1 ms here), writes the status word
    and returns; the host turns the word into a RuntimeError, clears it, and the next GEMM on the same context is
    correct.  No trap, no endless loop, no fault."""
    lib = _lib.load()
    ws = ops.status_word(cuda_dev)
    ops.check_device_status(cuda_dev)
    rc = lib.pq_wait_probe(ws.data_ptr(), ws.numel() * 4, 1000, torch.cuda.current_stream(cuda_dev).cuda_stream)
    assert rc == 0
    with pytest.raises(RuntimeError, match="wait gave up"):
        ops.check_device_status(cuda_dev)
    ops.check_device_status(cuda_dev)                               # the word was cleared by the read above
    run_gemm_case(cuda_dev, 300, 512, 256, lowrank=True, bias=True, seed=5)
    run_gemm_case(cuda_dev, 2049, 768, 384, lowrank=False, bias=True, seed=6)



@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("M,K,N", [(1, 128, 4), (127, 256, 60), (129, 128, 68), (300, 384, 1096), (260, 640, 132)])
def test_gemm_g32_tile_widths(cuda_dev, M, K, N, variant):
    """Both tile widths of the group-32 GEMM (and the choice by size) at the edges of their tiles and on ragged outputs."""
    g = torch.Generator().manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g).to(torch.float16)
    w = torch.randn(N, K, generator=g) * 0.02
    bias = torch.randn(N, generator=g) * 0.01
    xq, sa = oracle.quant_rows_g32(x)
    wq, sw = oracle.quant_rows_g32(w)
    _lib.set_option("g32_variant", variant)
    try:
        y = int8_exec.int8_gemm_g32(xq.to(cuda_dev), sa.to(cuda_dev), wq.to(cuda_dev), sw.t().contiguous().to(cuda_dev),
                                    bias.to(cuda_dev), torch.float16)
    finally:
        _lib.set_option("g32_variant", 0)
    assert torch.equal(y.cpu(), oracle.gemm_g32(xq, sa, wq, sw, bias, torch.float16))


# ------------------------------------------------------------------------------------------------ quantisation + down-projection
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,K1", [(1, 64, 0), (63, 128, 0), (64, 200, 0), (65, 1288, 0), (200, 1536, 0), (130, 1544, 0),
                                    (1000, 3072, 0), (9473, 3072, 0), (700, 6152, 0), (513, 12288, 0), (1300, 15360, 0),
                                    (96, 16384, 0), (2600, 192, 0), (130, 64, 8), (700, 3072, 12288), (5000, 1024, 520)])
def test_quant_rows_lowrank(cuda_dev, M, K, K1, dtype):
    """Codes and scales equal the quantiser's bit for bit; t lies within one unit in the last place of the fp64 product (plus
    the bound of an fp32 summation in any order).  Row and K tails, strided rows, slices of the last CTA that are short or
    empty, one to eight CTAs per row block, several blocks per CTA, two sources."""
    g = torch.Generator().manual_seed(M + K + K1)
    Kt = K + K1
    xp = torch.randn(M, Kt + 16, generator=g)
    xp[:, torch.randperm(Kt, generator=g)[: max(1, Kt // 200)]] *= 20.0
    xp = xp.to(dtype)
    x = xp[:, :Kt].contiguous()
    if M > 3:
        xp[2].zero_(); x[2].zero_()
    A = (torch.randn(Kt, 32, generator=g) * 0.05).to(dtype)
    a_t = A.t().contiguous().to(cuda_dev)
    xd = xp.to(cuda_dev)
    x0, x1 = xd[:, :K], xd[:, K:Kt] if K1 else None
    if K1 and x1.data_ptr() % 16:
        x1 = x1.contiguous()
    q, s, t = ops.quant_rows_lowrank(x0, a_t, x1)
    qs, ss = int8_exec.quant_rows(x.to(cuda_dev))
    assert torch.equal(q, qs) and torch.equal(s, ss)
    ref = x.to(cuda_dev).double() @ A.to(cuda_dev).double()
    mag = x.to(cuda_dev).double().abs() @ A.to(cuda_dev).double().abs()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    err = (t.double() - ref).abs()
    assert bool((err <= ulp * ref.abs() * 1.01 + 1e-6 * mag).all()), err.max().item()
    if Kt >= 512 and not K1:
        assert torch.equal(t, ops.lowrank_down(x0, a_t))              # the same slices, summed in the same order
        assert torch.equal(t[: M // 2], ops.quant_rows_lowrank(x0[: M // 2], a_t)[2])   # whatever the number of rows


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,K1", [(2500, 512, 0), (40, 1536, 0), (3001, 1544, 0), (40, 3072, 0), (1536, 3072, 0), (1537, 3072, 0),
                                    (9700, 3072, 0), (130, 6152, 0), (4200, 6152, 0), (2200, 12288, 0), (9700, 15360, 0),
                                    (4800, 16384, 0), (300, 16392, 0), (700, 3072, 6144), (5000, 1024, 520), (5000, 192, 72)])
def test_lowrank_down_is_one_sum_in_every_kernel(cuda_dev, M, K, K1, dtype):
    """t of a row is the same bits from the streaming kernel (many rows), from the cluster kernel (few long rows) and from the
    one-launch quantisation + down-projection, whatever the number of rows, for one source and for two; a last column slice
    that is short or missing, one to eight slices, rows beyond the one-launch form's length."""
    g = torch.Generator(device="cuda").manual_seed(M + K + K1)
    Kt = K + K1
    x = torch.randn(M, Kt, generator=g, device=cuda_dev).to(dtype)
    a_t = (torch.randn(32, Kt, generator=g, device=cuda_dev) * 0.05).to(dtype)
    t = ops.lowrank_down(x, a_t)
    if Kt <= 16384:
        assert torch.equal(t, ops.quant_rows_lowrank(x, a_t)[2])
    assert torch.equal(t[:33], ops.lowrank_down(x[:33], a_t)) and torch.equal(t[7:], ops.lowrank_down(x[7:], a_t))
    if K1:
        x0, x1 = x[:, :K].contiguous(), x[:, K:].contiguous()
        assert torch.equal(t, ops.lowrank_down_cat(x0, x1, a_t)) and torch.equal(t, ops.quant_rows_lowrank(x0, a_t, x1)[2])
        assert torch.equal(t[:33], ops.lowrank_down_cat(x0[:33], x1[:33], a_t))
    ref, mag = x.double() @ a_t.double().t(), x.double().abs() @ a_t.double().abs().t()
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert bool(((t.double() - ref).abs() <= ulp * ref.abs() * 1.01 + 1e-6 * mag).all())
    ops.check_device_status(cuda_dev)


# ------------------------------------------------------------------------------------------------ whole forward in one call
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N,lowrank", [(1, 64, 8, False), (154, 640, 1280, False), (77, 1808, 2376, False),
                                           (33, 512, 264, True), (700, 3072, 512, True)])
def test_linear_in_one_call(cuda_dev, M, K, N, lowrank, dtype):
    """`Int8Linear.forward` through the one-call entry point == the separate operators, bit for bit; also on a row-strided
    view, after a copy of the module, and after its scale buffer was replaced."""
    import copy
    g = torch.Generator().manual_seed(M + K + N)
    m = _toy_layer(cuda_dev, g, K, N, lowrank=lowrank, dtype=dtype)
    wide = rand_act(M, K + 24, dtype, M + 7).to(cuda_dev)
    for x in (wide[:, :K].contiguous(), wide[:, :K]):
        y = m(x)
        assert "_lean_cache" in m.__dict__
        xq, sx = int8_exec.quant_rows(x)
        if lowrank:
            want = int8_exec.int8_gemm_lr(xq, sx, m.weight_int8, m.w_scale, m.bias, m._down(x), m.lr_B, dtype)
        else:
            want = int8_exec.int8_gemm_fused(xq, sx, m.weight_int8, m.w_scale, m.bias, dtype)
        assert torch.equal(y, want)
    c = copy.deepcopy(m)
    assert torch.equal(c(x), want)
    c.w_scale = c.w_scale * 2
    assert torch.equal(m(x), want) and not torch.equal(c(x), want)
    # a bias and a branch that are set as plain attributes of a layer made without them take part
    if K % 32 == 0 and K >= 512 and N % 8 == 0:
        bare = _toy_layer(cuda_dev, g, K, N, lowrank=False, bias=False, dtype=dtype)
        bare.bias = torch.randn(N, generator=g).to(cuda_dev)
        with_bias = bare(x)
        assert torch.equal(with_bias, int8_exec.int8_gemm_fused(xq, sx, bare.weight_int8, bare.w_scale, bare.bias, dtype))
        bare.lr_A = (torch.randn(K, 32, generator=g) * 0.05).to(dtype).to(cuda_dev)
        bare.lr_B = (torch.randn(32, N, generator=g) * 0.05).to(dtype).to(cuda_dev)
        assert torch.equal(bare(x), int8_exec.int8_gemm_lr(xq, sx, bare.weight_int8, bare.w_scale, bare.bias, bare._down(x),
                                                           bare.lr_B, dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K", [(1, 32), (70, 256), (70, 480), (70, 512), (70, 16384), (70, 16416)])
def test_linear_fast_path_at_every_row_length(cuda_dev, M, K, dtype):
    """A rank-32 layer takes the fast path whether or not its down-projection shares the quantisation's launch (rows of 512 to
    16384 features), bit-equal to the separate operators, also on a row-strided input."""
    g = torch.Generator().manual_seed(M + K)
    N = 264
    m = _toy_layer(cuda_dev, g, K, N, lowrank=True, dtype=dtype)
    wide = rand_act(M, K + 24, dtype, M + 11).to(cuda_dev)
    for x in (wide[:, :K].contiguous(), wide[:, :K]):
        y = m(x)
        assert "_lean_cache" in m.__dict__
        xq, sx = int8_exec.quant_rows(x)
        assert torch.equal(y, int8_exec.int8_gemm_lr(xq, sx, m.weight_int8, m.w_scale, m.bias, m._down(x), m.lr_B, dtype))
    ops.check_device_status(cuda_dev)


class _Doubled(nn.Module):
    def forward(self, t):
        return t * 2

    def right_inverse(self, t):
        return t / 2


@pytest.mark.parametrize("where", ["parameter", "parametrised", "buffer"])
@pytest.mark.parametrize("names", [("bias",), ("lr_A", "lr_B"), ("w_scale",), ("weight_int8",), ("bias", "lr_A", "lr_B", "w_scale")])
def test_linear_operands_wherever_the_module_keeps_them(cuda_dev, names, where):
    """A layer's tensors take part in `forward` as `self.<name>` gives them, also after they became Parameters (an assignment
    or `load_state_dict(assign=True)`) or were parametrised: bit-equal to the separate operators and to `forward_into`, which
    reads the attributes."""
    g = torch.Generator().manual_seed(len(names))
    M, K, N, dtype = 70, 512, 264, torch.bfloat16
    m = _toy_layer(cuda_dev, g, K, N, lowrank="lr_A" in names, bias="bias" not in names, dtype=dtype)
    x = rand_act(M, K, dtype, 3).to(cuda_dev)
    before = m(x)
    for n in names:
        t = torch.randn(N, generator=g).to(cuda_dev) if n == "bias" else getattr(m, n).clone()
        if where == "buffer":
            if n == "bias":
                del m.bias
                m.register_buffer("bias", t)
            else:
                setattr(m, n, t)
        elif where == "parameter" or not t.is_floating_point():
            setattr(m, n, nn.Parameter(t, requires_grad=t.is_floating_point()))
        else:
            if n == "bias":
                m.bias = nn.Parameter(t)
            from torch.nn.utils import parametrize
            parametrize.register_parametrization(m, n, _Doubled(), unsafe=True)
    y = m(x)
    xq, sx = int8_exec.quant_rows(x)
    if m.lr_A is not None:
        want = int8_exec.int8_gemm_lr(xq, sx, m.weight_int8, m.w_scale, m.bias, m._down(x), m.lr_B, dtype)
    else:
        want = int8_exec.int8_gemm_fused(xq, sx, m.weight_int8, m.w_scale, m.bias, dtype)
    assert torch.equal(y, want)
    assert torch.equal(m.forward_into(x, torch.empty_like(y)), want)
    assert ("bias" in names) == (not torch.equal(y, before))


def test_linear_refuses_operands_that_do_not_fit(cuda_dev):
    """The library gets bare pointers, so a factor, scale or bias of another extent or device is an AssertionError before
    anything is launched; a strided bias is read through its strides."""
    g = torch.Generator().manual_seed(9)
    M, K, N, dtype = 70, 576, 264, torch.bfloat16
    x = rand_act(M, K, dtype, 4).to(cuda_dev)
    rnd = lambda *s: (torch.randn(*s, generator=g) * 0.05).to(dtype).to(cuda_dev)
    bad = [("lr_A", rnd(K - 64, 32)), ("lr_A", rnd(K + 64, 32)), ("lr_A", rnd(K, 32).cpu()), ("lr_B", rnd(32, N - 8)),
           ("lr_B", rnd(32, N).cpu()), ("w_scale", torch.rand(N - 8, device=cuda_dev)), ("w_scale", torch.rand(N)),
           ("bias", torch.rand(N + 8, device=cuda_dev)), ("bias", torch.rand(N)),
           ("weight_int8", torch.zeros(N - 8, K, dtype=torch.int8, device=cuda_dev))]
    for warm in (False, True):
        for name, t in bad:
            m = _toy_layer(cuda_dev, g, K, N, lowrank=True, dtype=dtype)
            if warm:
                m(x)
            setattr(m, name, t)
            with pytest.raises(AssertionError):
                m(x)
    m = _toy_layer(cuda_dev, g, K, N, lowrank=True, dtype=dtype)
    want = m(x)
    m.bias = torch.stack([m.bias, m.bias + 1], dim=1)[:, 0]
    assert not m.bias.is_contiguous() and torch.equal(m(x), want)


# ------------------------------------------------------------------------------------------------ out-of-place fusion
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hw,C,halo,boxes", [((32, 32), 64, 2, [(0, 16, 0, 32), (16, 32, 16, 48), (48, 64, 0, 16)]),
                                             ((17, 9), 8, 1, [(0, 2, 0, 2)]), ((8, 8), 3072, 0, [(0, 16, 0, 16)]),
                                             ((24, 40), 264, 3, [(40, 48, 72, 80), (0, 8, 0, 8)])])
def test_fuse_rows_out_of_place(cuda_dev, dtype, hw, C, halo, boxes):
    """`fuse_rows` in one launch == the in-place scatter on a clone, bit for bit, on contiguous and row-strided backgrounds:
    untouched rows (signed zeros included) go over as they are, the background itself is left alone; whole canvas covered,
    a single patch, patches at both ends of the token list."""
    g = torch.Generator().manual_seed(C + halo)
    H, W = hw
    plan = routing.build_route_plan(hw, boxes, halo, dtype=dtype)
    wide = torch.randn(1, H, W, C + 8, generator=g).to(dtype)
    wide[0, H - 1, W - 1] = -0.0
    y = torch.randn(plan.n_rows, C, generator=g).to(dtype).to(cuda_dev)
    for bg in (wide[..., :C].contiguous().to(cuda_dev), wide.to(cuda_dev)[..., :C]):
        before = bg.clone()
        want = bg.reshape(H * W, C).clone().contiguous()
        routing.scatter_rows_(y, plan, want)
        got = routing.fuse_rows(bg, y, plan)
        assert got.shape == (1, H, W, C)
        assert torch.equal(got.reshape(H * W, C).view(torch.int16), want.view(torch.int16))
        assert torch.equal(bg, before)


@pytest.mark.parametrize("extra", [[-1], [64, 2 ** 30], [5], [-3, 5, 64]])
def test_fuse_rows_with_a_hand_made_token_list(cuda_dev, extra):
    """Tokens outside the canvas are skipped and a token listed twice is blended as the in-place scatter blends it; every other
    row is the background's."""
    tokens = np.array([3, 5, 40] + extra, np.int32)
    n = tokens.size
    beta = np.full(n, 0.5, np.float32)
    plan = routing.RoutePlan(token_hw=(8, 8), patches=[], bucket_shapes=[], row_idx=np.arange(n, dtype=np.int32), m_hi=n,
                             tokens=tokens, ptr=np.arange(n + 1, dtype=np.int32), src=np.arange(n, dtype=np.int32), beta=beta)
    if extra.count(5):                                    # twice in one launch: the order is open, so both do the same
        plan.beta[:] = 1.0
        plan.src[:] = 0
    g = torch.Generator().manual_seed(n)
    bg = torch.randn(1, 8, 8, 64, generator=g).to(torch.bfloat16).to(cuda_dev)
    y = torch.randn(n, 64, generator=g).to(torch.bfloat16).to(cuda_dev)
    want = bg.reshape(64, 64).clone()
    inside = [i for i, t in enumerate(tokens) if 0 <= t < 64]
    routing.scatter_rows_(y, routing.RoutePlan(
        token_hw=(8, 8), patches=[], bucket_shapes=[], row_idx=plan.row_idx, m_hi=n, tokens=tokens[inside],
        ptr=np.arange(len(inside) + 1, dtype=np.int32), src=plan.src[inside], beta=plan.beta[inside]), want)
    torch.empty(64, 64, dtype=torch.bfloat16, device=cuda_dev).fill_(float("nan"))     # what a row left unwritten would hold
    assert torch.equal(routing.fuse_rows(bg, y, plan).reshape(64, 64), want)
    canvas = bg.reshape(64, 64).clone()
    assert torch.equal(routing.scatter_rows_(y, plan, canvas), want)


def test_fuse_rows_keeps_the_background_in_the_graph(cuda_dev):
    """The result carries the background's gradient and its forward-mode tangent, as a clone of it does; the values are those of
    an untracked background."""
    import torch.autograd.forward_ad as fwad
    plan = routing.build_route_plan((8, 8), [(0, 4, 0, 4)], 1)
    g = torch.Generator().manual_seed(5)
    bg = torch.randn(1, 8, 8, 64, generator=g).to(torch.bfloat16).to(cuda_dev)
    y = torch.randn(plan.n_rows, 64, generator=g).to(torch.bfloat16).to(cuda_dev)
    want = routing.fuse_rows(bg, y, plan)
    tracked = bg.clone().requires_grad_()
    got = routing.fuse_rows(tracked, y, plan)
    assert got.requires_grad and torch.equal(got.detach(), want)
    got.sum().backward()
    assert torch.equal(tracked.grad, torch.ones_like(bg))
    with torch.no_grad():
        assert torch.equal(routing.fuse_rows(tracked, y, plan), want)
    with fwad.dual_level():
        dual = fwad.make_dual(bg, torch.ones_like(bg))
        out = fwad.unpack_dual(routing.fuse_rows(dual, y, plan))
        assert torch.equal(out.primal, want) and out.tangent is not None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,K1", [(70, 512, 0), (1025, 736, 0), (300, 1536, 0), (300, 1568, 0), (130, 640, 384)])
def test_quant_rows_lowrank_under_capture(cuda_dev, M, K, K1, dtype):
    """Codes, scales and t recorded in a graph (few short rows: as two kernels) are those of the eager call (one kernel), and a
    replay reads the rows anew; one and two sources, a row length on either side of the line; the layer's forward as well."""
    g = torch.Generator().manual_seed(M + K)
    Kt = K + K1
    x = rand_act(M, Kt, dtype, M).to(cuda_dev)
    other = rand_act(M, Kt, dtype, M + 1).to(cuda_dev)
    m = _toy_layer(cuda_dev, g, Kt, 264, lowrank=True, dtype=dtype)
    a_t = m._lr_At()
    parts = (lambda v: (v[:, :K].contiguous(), v[:, K:].contiguous())) if K1 else (lambda v: (v, None))
    want = []
    for v in (x, other):
        x0, x1 = parts(v)
        want.append((*ops.quant_rows_lowrank(x0, a_t, x1), m(v)))
    x0, x1 = parts(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = (*ops.quant_rows_lowrank(x0, a_t, x1), m(x))
    for v, w in zip((x.clone(), other), want):
        x.copy_(v)
        if K1:
            x0.copy_(v[:, :K]); x1.copy_(v[:, K:])
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, w))
    ops.check_device_status(cuda_dev)


# ------------------------------------------------------------------------------------------------ several streams
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_layers_on_two_streams(cuda_dev, dtype):
    """Two layers whose forwards overlap on two streams (clusters of several CTAs next to the pair kernel, scratch of both from
    the allocator) give what they give one after the other, call after call."""
    g = torch.Generator().manual_seed(12)
    layers = [_toy_layer(cuda_dev, g, 3072, 1536, lowrank=True, dtype=dtype), _toy_layer(cuda_dev, g, 12288, 768, lowrank=True, dtype=dtype)]
    xs = [[rand_act(m_rows, m.in_features, dtype, 40 + i).to(cuda_dev) for i, m_rows in enumerate((900, 2100, 70))] for m in layers]
    want = [[m(x) for x in rows] for m, rows in zip(layers, xs)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(cuda_dev) for _ in layers]
    got = [[], []]
    for _ in range(8):
        for i in range(3):
            for j, (m, st) in enumerate(zip(layers, streams)):
                with torch.cuda.stream(st):
                    got[j].append((i, m(xs[j][i])))
    torch.cuda.synchronize()
    for j in range(2):
        assert all(torch.equal(y, want[j][i]) for i, y in got[j])
    ops.check_device_status(cuda_dev)


def test_host_row_pipeline(cuda_dev):
    """Pinned host rows in and out, two layers' pipelines enqueued before either is awaited: every row as the layer alone
    computes it, a last chunk that is short, repeated on the same buffers."""
    from pyraquant_b200.host_pipeline import HostRowPipeline
    g = torch.Generator().manual_seed(13)
    M, chunk, dtype = 1000, 384, torch.bfloat16
    layers = [_toy_layer(cuda_dev, g, 3072, 1024, lowrank=True), _toy_layer(cuda_dev, g, 6144, 512, lowrank=True)]
    hx = [rand_act(M, m.in_features, dtype, 50 + i).pin_memory() for i, m in enumerate(layers)]
    hy = [torch.full((M, m.out_features), float("nan"), dtype=dtype).pin_memory() for m in layers]
    pipes = [HostRowPipeline(m, m.in_features, dtype, cuda_dev, chunk) for m in layers]
    want = [torch.cat([m(x[a:a + chunk].to(cuda_dev)) for a in range(0, M, chunk)]).cpu() for m, x in zip(layers, hx)]
    for _ in range(3):
        for y in hy:
            y.fill_(float("nan"))
        for p, x, y in zip(pipes, hx, hy):
            p.start(x, y)
        for p in pipes:
            p.finish()
        assert all(torch.equal(y, w) for y, w in zip(hy, want))
    ops.check_device_status(cuda_dev)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quant_rows_with_infinities(cuda_dev, dtype):
    """Outside parity, but fixed: a row holding an infinity gets scale NaN and code -1 throughout, a NaN stays in its own row, and
    the neighbours are what they are without them; the one-launch prologue does the same."""
    x = rand_act(70, 1024, dtype, 77)
    clean = x.clone()
    x[3, 5], x[64, 1000], x[69, 0] = float("inf"), float("-inf"), float("nan")
    a_t = torch.zeros(32, 1024, dtype=dtype, device=cuda_dev)
    rows = [r for r in range(70) if r not in (3, 64, 69)]
    for q, s in (int8_exec.quant_rows(x.to(cuda_dev)), ops.quant_rows_lowrank(x.to(cuda_dev), a_t)[:2]):
        qo, so = oracle.quant_rows(clean)
        assert torch.equal(q.cpu()[rows], qo[rows]) and torch.equal(s.cpu()[rows], so[rows])
        assert bool(s[[3, 64]].isnan().all()) and bool((q[[3, 64]] == -1).all())
