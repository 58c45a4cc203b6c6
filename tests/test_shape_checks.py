"""Outputs of the wrong shape, type or layout are refused before anything is queued or written: the kernels and the
host threads get bare pointers, so nothing behind these checks could tell.  Every refused case raises on the host, before
CUDA is initialised, so those tests need no GPU."""
import numpy as np
import pytest
import torch

from trak_b200 import mmap_io
from trak_b200 import score_computers as sc

N, K, M = 40, 16, 6
BAD = [(N - 1, M), (N, M - 1), (N, M + 1), (0, M), (N, 1), (N,), (N, M, 1)]


@pytest.mark.parametrize("device", ["cpu", "meta"])
@pytest.mark.parametrize("shape", BAD)
def test_accumulators_that_do_not_hold_the_scores_are_refused(shape, device):
    computer = sc.B200ScoreComputer(torch.float32, "cuda:0")
    features, targets = torch.zeros(N, K), torch.zeros(M, K)
    acc = torch.zeros(shape, device=device)
    with pytest.raises(RuntimeError, match="accumulator"):
        computer.get_scores(features, targets, acc)
    with pytest.raises(RuntimeError, match="accumulator"):
        computer.get_scores_from_grads(features, torch.eye(K), targets, acc)


def test_too_few_row_weights_are_refused():
    computer = sc.B200ScoreComputer(torch.float32, "cuda:0")
    with pytest.raises(RuntimeError, match="row_scale"):
        computer.get_scores(torch.zeros(N, K), torch.zeros(M, K), torch.zeros(N, M), row_scale=torch.ones(N - 1))


@pytest.mark.parametrize("n, m, shape", [(N, M, (N, M)), (N, M, (N + 3, M)), (N, 1, (N, 5)), (0, M, (0, M))])
def test_what_torch_would_add_is_accepted(n, m, shape):
    sc._check_accumulator(n, m, torch.zeros(shape), None)


@pytest.mark.parametrize("out", [torch.zeros(7, 5), torch.zeros(8, 4), torch.zeros(8, 6), torch.zeros(8, 5).half(),
                                 torch.zeros(5, 8).T, torch.zeros(40)])
def test_outputs_of_a_product_have_its_shape(out):
    with pytest.raises(RuntimeError, match="out must be"):
        sc._check_out(out, 8, 5, torch.device("cpu"))
    sc._check_out(torch.zeros(8, 9)[:, 2:7], 8, 5, torch.device("cpu"))
    sc._check_out(torch.zeros(1, 8).T, 8, 1, torch.device("cpu"))


@pytest.mark.parametrize("dst", [np.zeros((3, 5), np.float32), np.zeros((4, 4), np.float32), np.zeros((4, 6), np.float32),
                                 np.zeros((4, 5), np.float16), np.zeros((4, 5), np.dtype(">f4")),
                                 np.zeros((4, 10), np.float32)[:, ::2], np.zeros((5, 4), np.float32).T,
                                 torch.zeros(3, 5), torch.zeros(4, 5).half(), torch.zeros(5, 4).T])
@pytest.mark.parametrize("add", [False, True])
def test_host_copies_go_to_arrays_of_the_same_shape_and_type(dst, add):
    with pytest.raises(ValueError, match="do not fit|cannot add|cannot copy|must be contiguous"):
        mmap_io.device_to_host(dst, torch.zeros(4, 5), object(), add=add)


def test_only_floats_are_added():
    with pytest.raises(ValueError, match="add"):
        mmap_io.device_to_host(torch.zeros(4, 5).half(), torch.zeros(4, 5).half(), object(), add=True)


def test_stores_opened_for_reading_are_not_written_to(tmp_path):
    mmap_io.create_store(tmp_path / "scores.mmap", (4, 5), torch.float32).flush()
    with pytest.raises(ValueError, match="read-only"):
        mmap_io.device_to_host(mmap_io.open_store(tmp_path / "scores.mmap", mode="r"), torch.zeros(4, 5), object())


@pytest.mark.parametrize("src", [np.zeros((4, 10), np.float32)[:, ::2], torch.zeros(5, 4).T])
def test_strided_host_sources_are_refused(src):
    with pytest.raises(ValueError, match="contiguous"):
        mmap_io.host_to_device(src, "cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["cuda", "cpu"])
@pytest.mark.parametrize("m, shape", [(M, (N + 3, M)), (1, (N, 5)), (1, (N + 2, 1))])
def test_scores_into_accumulators_that_torch_would_take(cuda, where, m, shape):
    gen = torch.Generator().manual_seed(m)
    features, targets = torch.randn(N, K, generator=gen), torch.randn(m, K, generator=gen)
    acc = torch.ones(shape, device=where)
    sc.B200ScoreComputer(torch.float32, cuda).get_scores(features, targets, acc)
    want = torch.ones(shape, dtype=torch.float64)
    want[:N] += features.double() @ targets.double().T
    assert torch.allclose(acc.double().cpu(), want, rtol=0, atol=1e-4)   # sums of 16 products of N(0, 1) values
    assert torch.equal(acc[N:].cpu(), torch.ones(shape)[N:])
