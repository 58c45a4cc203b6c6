"""How many host threads share a transfer: as many as the user of the process asks for, and which ones is not a secret."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "trak_b200", "libtrakb200.so")
ASK = """
import ctypes
lib = ctypes.CDLL({lib!r})
team = ctypes.c_int(-1)
print(lib.tb_host_threads(ctypes.byref(team)), team.value)
"""


def _run(code, threads=None):
    env = {k: v for k, v in os.environ.items() if k != "OMP_NUM_THREADS"}
    if threads is not None:
        env["OMP_NUM_THREADS"] = threads
    p = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert p.returncode == 0, p.stderr
    return tuple(int(v) for v in p.stdout.split()[-2:])


@pytest.mark.parametrize("threads, want", [("1", (1, 0)), ("3", (3, 0))])
def test_without_an_openmp_runtime(threads, want):
    assert _run(ASK.format(lib=LIB), threads) == want


def test_default_without_an_openmp_runtime():
    cores = len(os.sched_getaffinity(0))
    assert _run(ASK.format(lib=LIB)) == (max(1, min(12, cores - 1)), 0)


@pytest.mark.parametrize("threads, want", [("1", (1, 1)), ("3", (3, 1))])
def test_with_torch(threads, want):
    assert _run("import torch" + ASK.format(lib=LIB), threads) == want
    assert _run("import torch\ntorch.set_num_threads(2)" + ASK.format(lib=LIB), threads) == (2, 1)


C_HOST = """
import ctypes, glob, os
import numpy as np
rt = ctypes.CDLL(glob.glob({cudart!r})[0])
lib = ctypes.CDLL({lib!r})
lib.tb_host_to_device.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t]
lib.tb_device_to_host.argtypes = lib.tb_host_to_device.argtypes + [ctypes.c_int]
n = 9_000_001
src, dst, p = np.random.default_rng(0).random(n, np.float32), np.ones(n, np.float32), ctypes.c_void_p()
assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(4 * n)) == 0
for add in (0, 1, 1):
    assert lib.tb_host_to_device(0, None, p, src.ctypes.data, 4 * n) == 0
    assert lib.tb_device_to_host(0, None, dst.ctypes.data, p, 4 * n, add) == 0
want = src + src
want += src
assert np.array_equal(dst, want)
assert rt.cudaFree(p) == 0
team = ctypes.c_int(-1)
print(lib.tb_host_threads(ctypes.byref(team)), team.value)
"""


@pytest.mark.gpu
@pytest.mark.parametrize("threads", ["1", "2", "7"])
def test_round_trip_of_a_process_without_openmp(cuda, threads):
    import torch
    site = os.path.dirname(os.path.dirname(torch.__file__))
    cudart = os.path.join(site, "nvidia", "cuda_runtime", "lib", "libcudart.so.*")
    assert _run(C_HOST.format(lib=LIB, cudart=cudart), threads) == (int(threads), 0)


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [1, 2, 5])
def test_round_trip_with_a_team_of(cuda, threads):
    import torch
    from trak_b200 import mmap_io
    before = torch.get_num_threads()
    torch.set_num_threads(threads)
    try:
        src = torch.rand(9_000_001)
        dev = mmap_io.host_to_device(src, cuda)
        dst = torch.empty_like(src)
        mmap_io.device_to_host(dst, dev)
        assert torch.equal(dst, src)
        mmap_io.device_to_host(dst, dev, add=True)
        assert torch.equal(dst, src + src)
    finally:
        torch.set_num_threads(before)
