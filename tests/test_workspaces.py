"""Scratch buffers when several threads queue work on one stream."""
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from trak_b200 import _lib


def test_a_buffer_has_one_user_at_a_time():
    kept, cpu = _lib.Workspaces(most_kept=3), torch.device("cpu")
    a, b = kept.take(cpu, 7, 1000), kept.take(cpu, 7, 1000)
    assert a.data_ptr() != b.data_ptr() and a.numel() >= 1000
    kept.give(cpu, 7, a)
    assert kept.take(cpu, 7, 1000) is a
    kept.give(cpu, 7, a)
    assert kept.take(cpu, 7, 2000).numel() >= 2000
    for stream in range(10):
        kept.give(cpu, stream, a)
    assert len(kept.kept) == 3 and kept.take(cpu, 9, 1) is a
    kept.clear()
    assert not kept.kept


@pytest.mark.gpu
def test_threads_on_one_stream(cuda):
    from trak_b200 import fast_jl
    from trak_b200 import score_computers as sc
    gen = torch.Generator(device=cuda).manual_seed(1)
    xs = [torch.randn(700 + i, 3000, device=cuda, generator=gen) for i in range(4)]
    y = torch.randn(300, 3000, device=cuda, generator=gen)

    def work(x):
        return fast_jl.project(x, 512, 3, 148, _lib.TB_RADEMACHER), sc.gemm_nt(x, y), sc.gram(x[:, :200].contiguous())
    want = [work(x) for x in xs]
    torch.cuda.synchronize()
    with ThreadPoolExecutor(4) as pool:
        for got in pool.map(work, xs * 8):
            assert any(all(torch.equal(g, w) for g, w in zip(got, ws)) for ws in want if ws[0].shape == got[0].shape)


@pytest.mark.parametrize("shape,matrix,segments", [  # bytes of the 16-bit operands and the partial sums
    ((0, 16, 124_439_808, 8192, 148), 4_059_776_000, 4_059_778_048),
    ((1, 32, 124_439_808, 2048, 148), 8_003_159_040, 8_003_161_088),
    ((2, 32, 11_173_962, 4096, 148), 792_921_088, 792_923_136),
    ((0, 1, 592_003, 512, 148), 19_399_680, 19_401_728),
    ((0, 272, 1_000_003, 1024, 148), 743_212_032, 743_214_080),
    ((0, 7, 131, 512, 7), 115_712, 117_760),
    ((0, 512, 2_097_169, 4096, 148), 3_394_765_824, 3_394_767_872),
])
def test_least_workspace(shape, matrix, segments):
    lib = _lib.lib()
    assert lib.tb_project_least_workspace_bytes(*shape, 0) == matrix <= lib.tb_project_workspace_bytes(*shape)
    assert lib.tb_project_least_workspace_bytes(*shape, 62) == segments <= lib.tb_project_segments_workspace_bytes(*shape, 62)
    assert lib.tb_project_least_workspace_bytes(*shape, -1) == 0


def test_a_buffer_is_no_larger_than_there_is_room_for(monkeypatch):
    kept, cpu, empty = _lib.Workspaces(), torch.device("cpu"), torch.empty
    assert kept.take(cpu, 1, 4000, (int, 1000)).numel() == 4000
    assert kept.take(cpu, 1, 1000, (int, 4000)).numel() == 1000   # one size is asked for: `least` is not above it
    monkeypatch.setattr(_lib.Workspaces, "room", staticmethod(lambda device: 2500))
    small = kept.take(cpu, 1, 4000, (int, 1000))
    assert small.numel() == 1000
    kept.give(cpu, 1, small)
    assert kept.take(cpu, 1, 4000, (int, 1000)) is small          # the least is there already
    kept.give(cpu, 1, empty(2000, dtype=torch.uint8))
    assert kept.take(cpu, 1, 4000, (int, 1000)).numel() == 4000   # room once the kept one is given up

    def fragmented(n, **kw):
        if n > 1000:
            raise torch.cuda.OutOfMemoryError
        return empty(n, **kw)
    monkeypatch.setattr(torch, "empty", fragmented)
    monkeypatch.setattr(_lib.Workspaces, "room", staticmethod(lambda device: 1 << 62))
    assert kept.take(cpu, 1, 4000, (int, 1000)).numel() == 1000
    with pytest.raises(torch.cuda.OutOfMemoryError):
        kept.take(cpu, 1, 4000)


@pytest.mark.gpu
def test_projections_ask_for_what_they_use(cuda, monkeypatch):
    """Gaussian and stored matrices for the least, and a Rademacher one runs in it where there is no room for more."""
    from trak_b200 import fast_jl
    B, F, N, T = 4, 592_003, 512, 148
    lib, sizes, take = _lib.lib(), [], fast_jl._workspaces.take
    least, wanted = lib.tb_project_least_workspace_bytes(0, B, F, N, T, 0), lib.tb_project_workspace_bytes(0, B, F, N, T)
    table = lib.tb_project_least_workspace_bytes(0, B, F, N, T, 2) - least
    assert least < wanted

    def noted(dev, stream, nbytes, smaller=None):
        sizes.append(nbytes)
        return take(dev, stream, nbytes, smaller)
    monkeypatch.setattr(fast_jl._workspaces, "take", noted)
    g = torch.randn(B, F, generator=torch.Generator().manual_seed(2)).half().to(cuda)
    parts = [g[:, :1000].contiguous(), g[:, 1000:].contiguous()]
    stored = fast_jl.StoredMatrix(F, N, 5, T, _lib.TB_RADEMACHER, dtype=torch.float16, device=cuda)
    bytes_out = fast_jl.project(g, N, 5, T, _lib.TB_RADEMACHER)
    fast_jl.project(g, N, 5, T, _lib.TB_NORMAL)
    fast_jl.project(g, N, 5, T, _lib.TB_RADEMACHER, matrix=stored)
    fast_jl.project_segments(parts, N, 5, T, _lib.TB_NORMAL)
    fast_jl.project_segments(parts, N, 5, T, _lib.TB_RADEMACHER, matrix=stored)
    assert sizes == [wanted, least, least, least + table, least + table]
    fast_jl._workspaces.clear()
    monkeypatch.setattr(_lib.Workspaces, "room", staticmethod(lambda device: wanted - 1))
    small_out = fast_jl.project(g, N, 5, T, _lib.TB_RADEMACHER)
    fast_jl._workspaces.clear()
    assert torch.equal(fast_jl.project_segments(parts, N, 5, T, _lib.TB_RADEMACHER), small_out)
    # 16-bit operands: chains of 63 stages of 16-feature steps drift by less than 252 * 2^-24 of a sum
    worst = ((small_out - bytes_out).norm(dim=1) / bytes_out.norm(dim=1)).max()
    assert 0 < worst <= 2e-5


def test_static_scratch_takes_what_fits_the_least_workspace():
    """By the least size, not by the one with byte operands.  Device 63 does not exist, so nothing is launched."""
    lib, limit, N, T = _lib.lib(), 32 << 20, 512, 148

    def rc(B, F):
        return lib.tb_project_static(63, None, 0x1000, 0, B, F, F, 0x2000, N, N, 0, T, 0, 1.0, 0)
    for B, F in ((16, 600_011), (16, 870_000), (4, 592_003)):   # larger with byte operands than the scratch, or not
        assert lib.tb_project_least_workspace_bytes(0, B, F, N, T, 0) <= limit and rc(B, F) not in (0, 9)
    assert lib.tb_project_workspace_bytes(0, 16, 600_011, N, T) > limit
    for B, F in ((16, 900_000), (128, 2_000_000)):
        assert lib.tb_project_least_workspace_bytes(0, B, F, N, T, 0) > limit and rc(B, F) == 9
