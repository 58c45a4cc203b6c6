"""Copies between pageable host memory and the device through the library's threads and pinned rings."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MB = 1 << 20


# one thread's share, a short chunk, whole chunks of the ring, more than the ring holds, ragged ends
@pytest.mark.parametrize("nbytes", [1, 4095, 128 * 1024 + 1, 512 * 1024, MB + 3, 8 * MB, 32 * MB + 5, 75 * MB + 1])
def test_round_trip(cuda, nbytes):
    from trak_b200 import mmap_io
    src = torch.randint(0, 256, (nbytes,), dtype=torch.uint8)
    dev = mmap_io.host_to_device(src, cuda)
    assert torch.equal(dev.cpu(), src)
    dst = torch.zeros_like(src)
    mmap_io.device_to_host(dst, dev)
    assert torch.equal(dst, src)


@pytest.mark.parametrize("n", [1, 1000, 32 * 1024 + 1, 9 * MB + 3])
def test_accumulate(cuda, n):
    from trak_b200 import mmap_io
    x, y = torch.randn(n), torch.randn(n)
    want = y + x
    mmap_io.device_to_host(y, x.to(cuda), add=True)
    assert torch.equal(y, want)


def test_threads_and_streams_share_the_rings(cuda):
    from trak_b200 import _lib, mmap_io
    errors = []

    def work(seed):
        try:
            x = np.random.default_rng(seed).standard_normal((3, MB + 7)).astype(np.float32)
            stream = torch.cuda.Stream(cuda)
            for _ in range(3):
                with torch.cuda.stream(stream):
                    back = np.empty_like(x)
                    mmap_io.device_to_host(back, mmap_io.host_to_device(x, cuda) * 2)
                if not np.array_equal(back, x * 2):
                    errors.append(seed)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    _lib.check(_lib.lib().tb_host_staging_release())
    work(9)   # the rings are made again
    assert not errors
