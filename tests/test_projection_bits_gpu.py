"""Rademacher batches of up to 32 rows on the integer tensor cores, against the fp64 oracle.

Their sums are exact up to one rounding per partial: at most 148 partials, each rounded to fp32 once and added up in fp32,
are within (1 + sqrt(148)) * 2^-24 < 1e-6 of the row's norm.  Elements below 2^-17 of their row's largest are rounded to
2^-28 of it, which over F of them adds at most 2^-29 sqrt(F) of the norm."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import jl_oracle as o
from trak_b200 import _lib

RAD = 0
TOL = 1e-6
DT = {"f16": torch.float16, "f32": torch.float32, "bf16": torch.bfloat16}


def as_numpy(t):
    return t.view(torch.uint16).numpy() if t.dtype == torch.bfloat16 else t.numpy()


def grid(B, F, N, T=148):
    out = (ctypes.c_uint32 * 8)()
    assert _lib.lib().tb_project_grid(B, F, N, T, RAD, 148, out) == 0
    return dict(zip(("columns", "groups", "ctas", "tiles", "per_cta", "bundles", "stages", "chain"), out))


def project(g, N, seed, T, **kw):
    from trak_b200 import fast_jl
    return fast_jl.project(g, N, seed, T, RAD, **kw)


def worst_row(out, ref):
    out, ref = np.asarray(out, np.float64), np.asarray(ref, np.float64)
    return float((np.linalg.norm(out - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-300)).max())


def check(g_cpu, N, seed, T, cuda, tol=TOL):
    """The first and last 32 columns and two groups between them."""
    groups = sorted({0, 5, N // 64, N // 32 - 1})
    out = project(g_cpu.to(cuda), N, seed, T).cpu().numpy()
    ref = o.project_column_groups(RAD, as_numpy(g_cpu), seed, T, groups, round_f16=g_cpu.dtype == torch.float32)
    cols = np.concatenate([np.arange(32 * q, 32 * q + 32) for q in groups])
    assert worst_row(out[:, cols], ref) <= tol


def test_route_and_workspace():
    """Small matrices, more rows and tiles of more than 32,768 stages keep the 16-bit operand; no CTA sums up more."""
    def bits(*a):  # an odd number of stages is rounded up only here
        return grid(*a)["stages"] % 2 == 0 and grid(*a)["chain"] == grid(*a)["stages"]
    assert bits(16, 592_003, 512) and bits(1, 592_003, 512)
    assert bits(24, 330_003, 1536) and not bits(24, 310_003, 1536) and not bits(24, 990_003, 1024)
    assert bits(32, 782_003, 1536) and not bits(32, 780_003, 1536) and not bits(33, 1_990_003, 1536)
    assert not bits(17, 592_003, 512) and not bits(16, 572_003, 512)
    assert bits(16, 64 * 32_767, 512, 1) and not bits(16, 64 * 32_769, 512, 1)
    for F, T in ((64 * 32_767, 1), (40_000_000, 20), (124_439_808, 148), (300_000_000, 148)):
        g = grid(16, F, 1024, T)
        assert g["per_cta"] * g["stages"] <= 32_768
    lib = _lib.lib()
    # four bytes an element instead of two
    assert lib.tb_project_workspace_bytes(0, 16, 1_000_003, 512, 148) >= 4 * 16 * 1_000_003
    assert lib.tb_project_workspace_bytes(0, 16, 100_003, 512, 148) < 4 * 16 * 100_003 + 148 * 16 * 512 * 4


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f16", "f32", "bf16"])
@pytest.mark.parametrize("B,F,N,T", [
    (16, 592_003, 512, 148),      # 63 stages a tile: one is added
    (1, 590_000, 512, 148),
    (8, 100_003, 3072, 148),
    (9, 100_003, 3072, 132),
    (16, 9_000, 33_792, 148),     # a tile of less than one stage
    (5, 18_945, 16_384, 148),     # the last tile is short
    (16, 2_097_088, 512, 1),      # one tile, as long as 32-bit sums allow
    (3, 131, 2_300_416, 7),
    (17, 330_003, 1536, 148),     # from here on four groups to a CTA, one CTA per SM
    (24, 40_009, 12_800, 148),    # a box and a half per tile: the half is padding
    (25, 782_003, 1536, 147),     # a last bundle of fewer tiles than groups
    (32, 590_017, 2048, 3),       # fewer tiles than groups
    (20, 219, 2_300_416, 7),
])
def test_parity(cuda, B, F, N, T, dt):
    g = torch.randn(B, F, generator=torch.Generator().manual_seed(F)).mul_(1e-2).to(DT[dt])
    check(g, N, 11, T, cuda)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f16", "f32", "bf16"])
def test_values_of_all_sizes(cuda, dt):
    """Rows of widely spread magnitudes, one that outweighs its row, a constant row, zeros, and the ends of the type's range."""
    F = 592_003
    gen = torch.Generator().manual_seed(4)
    x = torch.randn(16, F, generator=gen)
    scale = torch.exp(3.0 * torch.randn(16, F, generator=gen))
    x[0] *= 1e-3 * scale[0]
    x[1] *= 1e-4
    x[1, 77] = 900.0
    x[2] = 0.37                                    # the sum of the entries is far above that of the signed ones
    x[3] = 0.0
    x[4] = 0.0
    x[4, F - 1] = 2.0 ** -24                       # the least fp16 number, alone in its row
    x[5] *= 2.0 ** -20                             # subnormal fp16 throughout
    x[6] *= 65504.0 / x[6].abs().max()
    x[7] *= 2.0 ** -120 if dt == "bf16" else 1.0   # bf16: products with 2^e need both factors
    x[8] *= 2.0 ** 112 if dt == "bf16" else 1.0    # their sums stay below 2^128
    x[9] *= 2.0 ** -133 if dt == "bf16" else 1.0   # subnormal bf16
    g = x.to(DT[dt])
    out = project(g.to(cuda), 512, 3, 148).cpu().numpy().astype(np.float64)
    ref = o.project(RAD, as_numpy(g), 512, 3, 148, round_f16=dt == "f32")
    rows = [b for b in range(16) if b not in (3, 4, 9)]
    assert worst_row(out[rows], ref[rows]) <= TOL + 2.0 ** -29 * F ** 0.5
    assert (out[3] == 0).all() and (out[4] == ref[4]).all()
    if dt == "bf16":   # fp32 results down to 2^-149: that much absolute
        assert np.abs(out[9] - ref[9]).max() <= 148 * 2.0 ** -149 + TOL * np.abs(ref[9]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f16", "f32", "bf16"])
def test_infinities_and_nan(cuda, dt):
    F, N = 592_003, 512
    g = torch.randn(6, F, generator=torch.Generator().manual_seed(1)).mul_(1e-2).to(DT[dt])
    inf = float("inf")
    g[0, 5] = inf
    g[1, 7], g[1, F - 1] = -inf, -inf
    g[2, 9], g[2, 400_000] = inf, -inf
    g[3, 11] = float("nan")
    g[4, 13], g[4, 14] = inf, float("nan")
    if dt == "f32":
        g[0, 5] = 1e6   # rounds to an fp16 infinity
    out = project(g.to(cuda), N, 5, 148).cpu().numpy()
    with np.errstate(invalid="ignore"):
        ref = o.project(RAD, as_numpy(g), N, 5, 148, round_f16=dt == "f32")
    assert (np.isnan(out) == np.isnan(ref)).all()
    assert (out[:3][np.isinf(ref[:3])] == ref[:3][np.isinf(ref[:3])]).all() and np.isinf(out[0]).all()
    assert worst_row(out[5:], ref[5:]) <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f16", "f32", "bf16"])
def test_segments_give_the_bits_of_the_dense_matrix(cuda, dt):
    """Parameters of odd widths, some of one element, strided and off any alignment; sums of integers in any order."""
    from trak_b200 import fast_jl
    widths = [1, 3, 392_001, 1, 511, 70_000, 129_487]
    F = sum(widths)
    g = torch.randn(12, F, generator=torch.Generator().manual_seed(2)).mul_(1e-2).to(DT[dt]).to(cuda)
    parts, at = [], 0
    for i, w in enumerate(widths):
        wide = torch.zeros(12, w + 5, dtype=g.dtype, device=cuda)
        wide[:, i % 4:i % 4 + w] = g[:, at:at + w]
        parts.append(wide[:, i % 4:i % 4 + w])
        at += w
    out = fast_jl.project_segments(parts, 512, 9, 148, RAD)
    assert torch.equal(out, project(g, 512, 9, 148))
    # a column slice of a wider buffer, 2 or 4 bytes off every alignment
    odd = torch.zeros(12, F + 3, dtype=g.dtype, device=cuda)
    odd[:, 1:F + 1] = g
    assert torch.equal(out, project(odd[:, 1:F + 1], 512, 9, 148, allow_strided=True))


@pytest.mark.gpu
def test_one_hot_rows_last_pass_accumulation_and_small_workspaces(cuda):
    F, N, T = 592_003, 512, 148
    feats = [0, 1, 15, 16, 4000, 4001, F - 1]
    hot = torch.zeros(len(feats), F, dtype=torch.float16, device=cuda)
    for i, f in enumerate(feats):
        hot[i, f] = 1.0
    assert (project(hot, N, 21, T).cpu().numpy() == o.matrix_rows(RAD, F, N, 21, T, feats)).all()
    # 256 rows with a 16-bit operand, the 16 behind them with bytes; into the same output, scaled
    g = torch.randn(272, F, generator=torch.Generator().manual_seed(3)).mul_(1e-2).half().to(cuda)
    out = torch.ones(272, N, device=cuda)
    project(g, N, 21, T, alpha=0.5, out=out, accumulate=True)
    last = project(g[256:], N, 21, T)
    assert torch.equal(out[256:], 0.5 * last + 1.0)
    assert worst_row(out[:256].cpu() - 1.0, 0.5 * o.project(RAD, g[:256].cpu().numpy(), N, 21, T)) <= 1e-4
    # the library's own scratch has no room for four bytes an element of these: accepted as before
    big = torch.randn(16, 600_011, generator=torch.Generator().manual_seed(5)).mul_(1e-2).half().to(cuda)
    lib, res = _lib.lib(), torch.empty(16, N, device=cuda)
    stream = torch.cuda.current_stream(cuda).cuda_stream
    assert lib.tb_project_workspace_bytes(0, 16, 600_011, N, T) > 32 << 20
    assert lib.tb_project_static(0, stream, big.data_ptr(), 0, 16, 600_011, 600_011, res.data_ptr(), N, N, 21, T, RAD,
                                 1.0, 0) == 0
    assert worst_row(res.cpu(), project(big, N, 21, T).cpu()) <= 1e-4


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f16", "f32", "bf16"])
@pytest.mark.parametrize("B,F,N", [(16, 592_003, 512), (24, 330_003, 1536)])
def test_rows_that_few_elements_outweigh(cuda, B, F, N, dt):
    """Elements of a step of the largest element's and less, up to the most that may outweigh the others, at both ends of the
    exponents.  Rounding may take 2^-24 of the largest element and 2^-22 of the norm of the rest."""
    gen = torch.Generator().manual_seed(6)
    x = torch.randn(B, F, generator=gen, dtype=torch.float64)
    u = torch.rand(F, generator=gen, dtype=torch.float64)
    top = 1.0 if dt == "bf16" else 2.0 ** 15        # fp16: steps of its least number reach 2^39 below
    x[0], x[0, 77] = (1 + u) * 2.0 ** -30 * top, top
    x[1], x[1, F - 1] = 2.0 ** -28 * top, top       # half a step each
    x[2], x[2, 5::50_021] = x[2] * 2.0 ** -16 * top, -top
    x[3], x[3, 0::997] = x[3] * 2.0 ** -24 * top, 2.0 ** -8 * top
    x[3, 40] = top
    x[4] = torch.exp(3 * x[4]) * torch.randn(F, generator=gen, dtype=torch.float64)
    x[4] *= top / x[4].abs().max()
    x[5], x[5, 4000:4016] = x[5] * 2.0 ** -20 * top, top                       # all of one place of a tile
    x[6], x[6, 9::8191] = torch.where(u < 0.01, x[6] * 2.0 ** -18 * top, torch.zeros(F, dtype=torch.float64)), top
    if dt == "bf16":
        x[7], x[7, 3] = (1 + u) * 2.0 ** 90, 2.0 ** 118
        x[8], x[8, 3] = (1 + u) * 2.0 ** -125, 2.0 ** -97
    g = x.to(DT[dt])
    check(g, N, 23, 148, cuda, tol=TOL + 2.0 ** -24 + 2.0 ** -22)
    # the parameters of a model, in the same bits
    from trak_b200 import fast_jl
    dense, cut = g.to(cuda), F // 3
    parts = [dense[:, :1].contiguous(), dense[:, 1:cut].contiguous(), dense[:, cut:].contiguous()]
    assert torch.equal(fast_jl.project_segments(parts, N, 23, 148, RAD), project(dense, N, 23, 148))
