"""Products and inverses at the sizes where the tile, the slices of the contraction and the block columns change."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


# one 128-wide tile and its neighbours, few tiles and a long contraction (sliced), a ragged last slice, rows longer
# than a warp, two, four, eight warps hold in registers and than one span of the packing kernel
@pytest.mark.parametrize("M,N,K", [(1, 1, 40), (127, 129, 32), (128, 128, 64), (257, 255, 4096), (100, 300, 8192),
                                   (513, 100, 1025), (64, 64, 2049), (40, 500, 4100), (33, 65, 9000), (1000, 512, 512)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_gemm_nt(cuda, M, N, K, dtype):
    from trak_b200 import score_computers as sc
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    a = torch.randn(M, K, device=cuda, generator=g).to(dtype)
    b = torch.randn(N, K, device=cuda, generator=g).to(dtype)
    w = torch.rand(M, device=cuda, generator=g)
    want = w.double()[:, None] * (a.double() @ b.double().T)
    got = sc.gemm_nt(a, b, row_scale=w)
    assert rel(got, want) <= 3e-5
    assert rel(sc.gemm_nt(a, b, out=got.clone(), row_scale=w, accumulate=True), 2 * want) <= 3e-5


@pytest.mark.parametrize("M", [65535 * 128, 65535 * 128 + 1])
def test_gemm_nt_of_more_rows_than_a_grid_of_small_tiles_has(cuda, M):
    from trak_b200 import score_computers as sc
    a = torch.randn(M, 8, device=cuda, generator=torch.Generator(device=cuda).manual_seed(M)).half()
    b = torch.randn(3, 8, device=cuda, generator=torch.Generator(device=cuda).manual_seed(8)).half()
    want = a.float() @ b.float().T
    assert rel(sc.gemm_nt(a, b), want.double()) <= 1e-6   # eight products of 11-bit numbers: nearly exact either way


@pytest.mark.parametrize("n,k", [(5000, 40), (4097, 129), (3001, 512), (20000, 300), (100, 700), (1, 5), (513, 17), (1030, 145),
                                 (2048, 300), (2049, 31)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_gram(cuda, n, k, dtype):
    from trak_b200 import score_computers as sc
    x = torch.randn(n, k, device=cuda, generator=torch.Generator(device=cuda).manual_seed(n)).to(dtype)
    want = x.double().T @ x.double()
    got = sc.gram(x)
    assert torch.equal(got, got.T)
    assert rel(got, want) <= (2e-6 if dtype == torch.float32 else 3e-5)
    got = sc.gram(x, out=got, accumulate=True)
    assert torch.equal(got, got.T) and rel(got, 2 * want) <= (2e-6 if dtype == torch.float32 else 3e-5)


@pytest.mark.parametrize("k", [1, 3, 4, 63, 65, 127, 130, 448, 449, 512, 575, 640, 1088])
def test_inverse_at_tile_edges(cuda, k):
    from trak_b200 import score_computers as sc
    y = torch.randn(3 * k, k, device=cuda, dtype=torch.float64, generator=torch.Generator(device=cuda).manual_seed(k))
    a = (y.T @ y / k).float()
    want = torch.linalg.inv(a.double() + 1e-3 * torch.eye(k, device=cuda, dtype=torch.float64))
    got = sc.spd_inverse_(a.clone(), 1e-3, rescale=False)
    assert rel(got, want) <= 2e-5
    wide = torch.zeros(k, k + 3, device=cuda)      # rows that are not 16-byte aligned
    wide[:, :k] = a
    assert rel(sc.spd_inverse_(wide[:, :k], 1e-3, rescale=False), want) <= 2e-5


@pytest.mark.parametrize("k", [1025, 1536, 1537, 2100, 2560, 3111])
def test_inverse_of_several_block_columns(cuda, k):
    """Columns, updates and merges run on three streams: the same bits from call to call and from several threads."""
    from concurrent.futures import ThreadPoolExecutor
    from trak_b200 import score_computers as sc
    y = torch.randn(2 * k, k, device=cuda, dtype=torch.float64, generator=torch.Generator(device=cuda).manual_seed(k))
    a = (y.T @ y / k).float()
    want = torch.linalg.inv(a.double() + 1e-2 * torch.eye(k, device=cuda, dtype=torch.float64))
    got = sc.spd_inverse_(a.clone(), 1e-2, rescale=False)
    assert rel(got, want) <= 2e-5
    assert torch.equal(got, got.T)
    torch.cuda.synchronize()

    def again(_):
        with torch.cuda.stream(torch.cuda.Stream()):
            out = [sc.spd_inverse_(a.clone(), 1e-2, rescale=False) for _ in range(3)]
            torch.cuda.current_stream().synchronize()
        return all(torch.equal(o, got) for o in out)
    with ThreadPoolExecutor(3) as pool:
        assert all(pool.map(again, range(3)))


@pytest.mark.parametrize("m, n, k", [(1, 1, 1), (129, 257, 33), (3000, 512, 1100)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_product_in_two_steps(cuda, m, n, k, dtype):
    from trak_b200 import score_computers as sc
    gen = torch.Generator(device=cuda).manual_seed(m + n)
    a = torch.randn(m, k, device=cuda, generator=gen).to(dtype)
    b = torch.zeros(n, k, device=cuda, dtype=dtype)
    values = torch.randn(n, k, device=cuda, generator=gen).to(dtype)
    scale = torch.rand(m, device=cuda, generator=gen)
    got = sc.gemm_nt(a, b, row_scale=scale, b_ready=lambda: b.copy_(values))
    assert torch.equal(got, sc.gemm_nt(a, values, row_scale=scale))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_features_of_a_matrix_packed_beside_the_inverse(cuda, monkeypatch, dtype):
    """A single block, on the caller's stream and packed on a stream of its own while the inverse is computed."""
    from trak_b200 import score_computers as sc
    asked, pair = [], sc.B200ScoreComputer._pair
    monkeypatch.setattr(sc.B200ScoreComputer, "_pair", lambda self, wanted: asked.append(wanted) or pair(self, wanted))
    x = torch.randn(5000, 1100, device=cuda, generator=torch.Generator(device=cuda).manual_seed(3)).to(dtype)
    computer = sc.B200ScoreComputer(dtype, cuda)
    xtx = computer.get_xtx(x)
    want = computer.get_x_xtx_inv(x, xtx)
    monkeypatch.setattr(sc.B200ScoreComputer, "APART_BYTES", 0)
    got = computer.get_x_xtx_inv(x, xtx)
    assert asked == [False, False, True]   # the Gram, then the features either way
    assert torch.equal(got, want)


@pytest.mark.parametrize("where", ["cuda", "cpu"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_one_plane_gram_of_many_rows(cuda, where, dtype):
    """A chain of n / 16 steps, each of which truncates below the last of 24 places, loses at most n / 16 * 2^-23; blocks
    of a host matrix, two partial sums and slices only shorten it."""
    from trak_b200 import score_computers as sc
    n, k = 50_000, 300
    x = torch.randn(n, k, device=cuda, generator=torch.Generator(device=cuda).manual_seed(5)).to(dtype)
    want = x.double().T @ x.double()
    got = sc.B200ScoreComputer(torch.float32, cuda).get_xtx(x.to(where))
    assert rel(got, want) <= n / 16 * 2.0 ** -23
