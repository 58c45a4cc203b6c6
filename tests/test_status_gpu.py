"""The status word on its way to the host: what a call takes from the driver for it, and whose status a read reports."""
import os
import subprocess
import sys
import threading
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

pytestmark = pytest.mark.gpu

B, F, N, TILES = 16, 50021, 1024, 148


def _call(lib, dev, name, g, out, ws=None, nbytes=None):
    stream = torch.cuda.current_stream(dev).cuda_stream
    args = [dev.index, stream, g.data_ptr(), 0, g.shape[0], g.shape[1], g.stride(0), out.data_ptr(), N, N, 17, TILES, 0,
            1.0, 0]
    if name == "tb_project":
        args += [ws.data_ptr(), ws.numel() if nbytes is None else nbytes]
    return getattr(lib, name)(*args)


@pytest.fixture
def job(cuda):
    from trak_b200 import _lib
    lib = _lib.lib()
    g = (torch.randn(B, F, device=cuda) * 1e-2).half()
    ws = torch.empty(lib.tb_project_workspace_bytes(0, B, F, N, TILES), dtype=torch.uint8, device=cuda)
    out = torch.empty(B, N, device=cuda)
    for name in ("tb_project", "tb_project_static"):   # the one-time set-up of this device, before any capture
        assert _call(lib, cuda, name, g, out, ws) == 0
    torch.cuda.synchronize()
    return lib, g, out, ws


@pytest.mark.parametrize("name", ["tb_project_static", "tb_project"])
def test_first_call_of_a_thread_can_be_captured(cuda, job, name):
    """A thread's first call allocates nothing: under a capture an allocation would be refused and end it.  (So no
    memory is left behind by threads that end, either.)"""
    lib, g, want, ws = job
    got, codes = torch.zeros_like(want), []
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream(cuda)
    torch.cuda.synchronize()

    def work():
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="global")
            try:
                codes.append(_call(lib, cuda, name, g, got, ws))
            finally:
                graph.capture_end()

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert codes == [0], lib.tb_last_cuda_error()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


FIRST_WORD = """
import torch
from trak_b200 import _lib
lib, dev = _lib.lib(), torch.device("cuda", 0)
g, out = (torch.randn(16, 50021, device=dev) * 1e-2).half(), torch.empty(16, 1024, device=dev)
ws = torch.empty(lib.tb_project_workspace_bytes(0, 16, 50021, 1024, 148), dtype=torch.uint8, device=dev)
def args():
    return [0, torch.cuda.current_stream().cuda_stream, g.data_ptr(), 0, 16, 50021, 50021, out.data_ptr(), 1024, 1024, 17,
            148, 0, 1.0, 0]
assert lib.tb_project_static(*args()) == 0
want = out.clone()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, capture_error_mode="global"):
    assert lib.tb_project(*args(), ws.data_ptr(), ws.numel()) == 0, lib.tb_last_cuda_error()
out.zero_()
graph.replay()
torch.cuda.synchronize()
assert torch.equal(out, want)
assert lib.tb_stream_status(0, torch.cuda.current_stream().cuda_stream, None) == 0
"""


def test_the_process_makes_its_words_under_a_capture(cuda):
    """tb_project_static makes no words, so the first ones may be wanted while a capture is going on."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", FIRST_WORD], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr


def test_a_word_that_was_handed_out_again_is_not_believed(cuda, job):
    """More reads than there are words between a call and its status: the status comes from the device then."""
    lib, g, out, ws = job
    own, other = torch.cuda.Stream(cuda), torch.cuda.Stream(cuda)
    torch.cuda.synchronize()
    with ThreadPoolExecutor(1) as pool, torch.cuda.stream(own):
        def call():
            with torch.cuda.stream(own):
                return _call(lib, cuda, "tb_project", g, out, ws)
        assert pool.submit(call).result() == 0
        for _ in range(1500):
            assert lib.tb_stream_status(cuda.index, other.cuda_stream, None) == 0
        assert pool.submit(lib.tb_stream_status, cuda.index, own.cuda_stream, None).result() == 0
        assert pool.submit(call).result() == 0
        for _ in range(1500):
            assert lib.tb_stream_status(cuda.index, other.cuda_stream, None) == 0
        assert lib.tb_selftest_wait_timeout(cuda.index, other.cuda_stream, 20) == 0
        other.synchronize()
        assert pool.submit(lib.tb_stream_status, cuda.index, own.cuda_stream, None).result() == 7
    assert lib.tb_stream_status(cuda.index, own.cuda_stream, None) == 0


def test_a_call_that_was_refused_does_not_vouch_for_the_device(cuda, job):
    """A wait runs out, then a projection is refused for its size: the status read after it reports the wait, and not
    the word that the last accepted call left."""
    lib, g, out, ws = job
    stream = torch.cuda.current_stream(cuda)
    assert _call(lib, cuda, "tb_project", g, out, ws) == 0
    assert lib.tb_stream_status(cuda.index, stream.cuda_stream, None) == 0
    assert lib.tb_selftest_wait_timeout(cuda.index, stream.cuda_stream, 20) == 0
    # 2^31 rows of 64 features and more do not fit a tensor map; the sizes are looked at before any pointer is used
    F, rows = 1 << 34, 16
    rc = lib.tb_project(cuda.index, stream.cuda_stream, g.data_ptr(), 0, rows, F, F, out.data_ptr(), N, N, 17, TILES, 0,
                        1.0, 0, ws.data_ptr(), 1 << 60)
    assert rc == 8, lib.tb_strerror(rc)
    assert lib.tb_stream_status(cuda.index, stream.cuda_stream, None) == 7
    assert lib.tb_stream_status(cuda.index, stream.cuda_stream, None) == 0


FIRST_READ = """
import torch
from trak_b200 import _lib
lib, other = _lib.lib(), torch.cuda.Stream()
stream = torch.cuda.current_stream().cuda_stream
assert lib.tb_selftest_wait_timeout(0, stream, 20) == 0     # before there is a word for kernels to repeat a failure in
assert lib.tb_stream_status(0, stream, None) == 7
assert lib.tb_stream_status(0, stream, None) == 0
for s in (stream, other.cuda_stream):                       # and with it, on either stream
    assert lib.tb_selftest_wait_timeout(0, s, 20) == 0
    assert lib.tb_stream_status(0, s, None) == 7
    assert lib.tb_stream_status(0, stream, None) == 0
    assert lib.tb_device_status(0, None) == 0
assert lib.tb_selftest_wait_timeout(0, stream, 20) == 0
assert lib.tb_device_status(0, None) == 7                   # read by the other call: nothing is left for the stream's
assert lib.tb_stream_status(0, stream, None) == 0
"""


def test_a_failure_reaches_the_first_read_of_a_process_and_the_later_ones(cuda):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", FIRST_READ], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr


FIRST_READ_UNDER_A_CAPTURE = """
import threading
import torch
from trak_b200 import _lib
lib = _lib.lib()
assert lib.tb_device_status(0, None) == 0   # the one-time set-up of the device
x, side = torch.zeros(8, device="cuda"), torch.cuda.Stream()
side.wait_stream(torch.cuda.current_stream())
graph, codes = torch.cuda.CUDAGraph(), []
torch.cuda.synchronize()
with torch.cuda.graph(graph, capture_error_mode="thread_local"):   # "global" forbids any thread's wait for a stream
    x.add_(1.0)
    t = threading.Thread(target=lambda: codes.append(lib.tb_stream_status(0, side.cuda_stream, None)))
    t.start()
    t.join()
    x.add_(1.0)
graph.replay()
torch.cuda.synchronize()
assert codes == [0] and x.tolist() == [2.0] * 8, (codes, x)
"""


def test_the_first_read_beside_another_threads_capture(cuda):
    """It makes its word on a stream of its own, so the capture goes on."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", FIRST_READ_UNDER_A_CAPTURE], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr


def test_a_call_answers_for_itself_and_leaves_a_later_failure_to_its_own_caller(cuda, job):
    """Thread A projects; then thread B's inverse, on a stream of its own, fails; A reads its status first."""
    lib, g, out, ws = job
    a, b = torch.cuda.Stream(cuda), torch.cuda.Stream(cuda)
    assert lib.tb_stream_status(cuda.index, b.cuda_stream, None) == 0   # kernels repeat failures to the host from here on
    indefinite = -torch.eye(64, device=cuda)
    scratch = torch.empty(lib.tb_spd_inverse_workspace_bytes(64), dtype=torch.uint8, device=cuda)
    torch.cuda.synchronize()
    with ThreadPoolExecutor(1) as thread_a, ThreadPoolExecutor(1) as thread_b:
        def project():
            with torch.cuda.stream(a):
                return _call(lib, cuda, "tb_project", g, out, ws)

        def invert():
            return lib.tb_spd_inverse(cuda.index, b.cuda_stream, indefinite.data_ptr(), 64, 64, 0.0, 0, None,
                                      scratch.data_ptr(), scratch.numel())

        def status(stream):
            return lib.tb_stream_status(cuda.index, stream.cuda_stream, None)
        assert thread_a.submit(project).result() == 0
        a.synchronize()
        assert thread_b.submit(invert).result() == 0
        b.synchronize()
        assert thread_a.submit(status, a).result() == 0
        assert thread_b.submit(status, b).result() == 10   # TB_ERR_NOT_SPD
        assert thread_b.submit(status, b).result() == 0
