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
