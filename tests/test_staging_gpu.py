"""Restaging of gradients that start at any byte: rows, tiles and parameters that are not 16-byte aligned."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles shorter than a run, of exactly one and two runs (256 fp32 or 512 16-bit features) and ragged beyond; pitches that
# move every row to another alignment
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("F,tiles", [(37, 4), (2048, 4), (4096, 4), (3001, 2), (5555, 3)])
@pytest.mark.parametrize("first,pitch_extra", [(0, 0), (1, 1), (2, 3), (3, 6), (7, 9)])
def test_views_equal_copies(cuda, dtype, F, tiles, first, pitch_extra):
    from trak_b200 import _lib, fast_jl
    wide = torch.randn(21, first + F + pitch_extra, device=cuda).to(dtype)
    view = wide[:, first:first + F]
    for ptype in (_lib.TB_RADEMACHER, _lib.TB_NORMAL):
        want = fast_jl.project(view.contiguous(), 512, 3, tiles, ptype)
        assert torch.equal(fast_jl.project(view, 512, 3, tiles, ptype, allow_strided=True), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("widths", [[1, 700, 3, 2049, 1], [513, 511, 1024], [5] * 300, [4000, 1, 1, 4000]])
def test_parameters_equal_their_concatenation(cuda, dtype, widths):
    from trak_b200 import _lib, fast_jl
    parts = [torch.randn(19, w, device=cuda).to(dtype) for w in widths]
    want = fast_jl.project(torch.cat(parts, 1), 512, 5, 3, _lib.TB_RADEMACHER)
    assert torch.equal(fast_jl.project_segments(parts, 512, 5, 3, _lib.TB_RADEMACHER), want)
