"""Score computer with the reference's interface, running on the sm_100a kernels.

Mirrors ``BasicScoreComputer`` (trak/score_computers.py:114-189): same constructor
arguments, same three methods, same shapes and dtypes of the results, so it can be
passed to an unmodified ``TRAKer(score_computer=B200ScoreComputer)``
(trak/traker.py:186-193).  Differences:

* products run on the tensor cores (fp32 inputs as row-scaled fp16 hi + lo planes, three
  passes; the Gram is accumulated 64 rows at a time, so it is as accurate as an fp32 GEMM);
* the regularised inverse goes through Cholesky in fp32 instead of LU and raises
  ``NotPositiveDefinite`` where the matrix is not positive definite;
* Gram blocks are accumulated in fp32 whatever ``dtype`` is (the reference adds
  them in ``dtype``) and cast once at the end;
* with a ``process_group`` the Gram of this rank's rows is summed over the group
  (one all-reduce of k x k fp32) -- rows sharded across GPUs, everything else
  local: the inverse is replicated, features and scores stay row-sharded;
* ``get_scores`` takes an optional ``row_scale`` (the out-to-loss weights) that is
  applied inside the GEMM epilogue, and streams the scores to a host accumulator while the
  next block is being multiplied.

There is no CPU path: tensors are moved to ``device`` and the CUDA library must load.
"""
import logging
import threading

import torch

from . import _lib, mmap_io

_DTYPES = {torch.float16: _lib.TB_F16, torch.bfloat16: _lib.TB_BF16, torch.float32: _lib.TB_F32}
_workspaces = _lib.Workspaces()
_pairs = threading.local()


def free_workspaces():
    _workspaces.clear()
    _lib.check(_lib.lib().tb_host_staging_release())


class StreamPair:
    """Two side streams that row blocks alternate between.  Every product here is a memory-bound packing pass
    (row maxima, fp16 hi / lo planes) followed by a tensor-core GEMM; on one stream the packing of block i + 1
    waits for the GEMM of block i although the two use different parts of the SM.  With blocks alternating
    between two streams the packing (and any host-to-device copy) of one block runs under the GEMM of the other.
    Inside ``with pair:`` a side stream waits for what the caller's stream had been given on entry, and the caller's
    stream waits on exit for the side streams that were used; ``with pair.stream(i):`` makes stream ``i % 2`` current.  Work that touches the same memory
    from consecutive blocks (an accumulator, a reused buffer) must be given one buffer per stream."""

    def __init__(self, device):
        self.device = torch.device(device)
        self.streams = [torch.cuda.Stream(self.device), torch.cuda.Stream(self.device)]
        self.entered, self.done = torch.cuda.Event(), [torch.cuda.Event(), torch.cuda.Event()]

    def __enter__(self):
        self.main = torch.cuda.current_stream(self.device)
        self.entered.record(self.main)
        self.used = [False, False]
        return self

    def __exit__(self, *exc):
        for s, done, used in zip(self.streams, self.done, self.used):
            if used:
                done.record(s)
                self.main.wait_event(done)
        return False

    def stream(self, i: int):
        s = self.streams[i % 2]
        if not self.used[i % 2]:
            self.used[i % 2] = True
            s.wait_event(self.entered)
        return torch.cuda.stream(s)

    def current(self, i: int):
        return self.streams[i % 2]

    def uses(self, t: torch.Tensor):
        """``t`` is used on the current stream, which may not be the one it was allocated on."""
        t.record_stream(torch.cuda.current_stream(self.device))

    def mark(self):
        """The point the current stream has reached, for ``after``."""
        event = torch.cuda.Event()
        event.record(torch.cuda.current_stream(self.device))
        return event

    def after(self, event):
        torch.cuda.current_stream(self.device).wait_event(event)


class OneStream:
    """Stands in for a ``StreamPair`` where there is one block only: everything stays on the caller's stream."""

    def __init__(self, device):
        self.device = device

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False

    def stream(self, i: int):
        return self

    def current(self, i: int):
        return torch.cuda.current_stream(self.device)

    def uses(self, t):
        pass

    def mark(self):
        pass

    def after(self, event):
        pass


def _as_device_matrix(t: torch.Tensor, device) -> torch.Tensor:
    if not t.is_cuda and t.dtype in _DTYPES and t.is_contiguous() and torch.device(device).type == "cuda" \
            and t.numel() * t.element_size() >= mmap_io.NATIVE_MIN_BYTES and not t.is_pinned():
        t = mmap_io.host_to_device(t, device)
    else:
        t = t.to(device, non_blocking=True)
    if t.dtype not in _DTYPES:
        t = t.float()
    if t.dim() != 2:
        raise RuntimeError("expected a 2-D tensor")
    if t.stride(1) != 1 or t.stride(0) < t.shape[1]:
        t = t.contiguous()
    return t


def _check_out(out: torch.Tensor, rows: int, cols: int, device) -> int:
    """The kernels write ``rows`` x ``cols`` floats from ``out``'s pointer on: anything else would be written past its
    end, or not where the caller looks.  Returns the rows' distance."""
    if out.shape != (rows, cols) or out.dtype != torch.float32 or out.device != device \
            or (cols > 1 and out.stride(1) != 1):
        raise RuntimeError(f"out must be a float32 [{rows}, {cols}] tensor with unit column stride on the operands' device")
    return out.stride(0)


def _check_accumulator(n: int, m: int, accumulator: torch.Tensor, row_scale) -> None:
    """Raises before anything is queued where ``accumulator += [n, m] scores`` is not defined.  Rows beyond ``n`` are
    left as they are; a single column of scores is added to every column, as torch's broadcasting has it."""
    if accumulator.dim() != 2 or accumulator.shape[0] < n or (accumulator.shape[1] != m and m != 1):
        raise RuntimeError(f"accumulator of shape {list(accumulator.shape)} does not hold [{n}, {m}] scores")
    if row_scale is not None and row_scale.numel() < n:
        raise RuntimeError("row_scale must have one entry per row of the features")


def gram(x: torch.Tensor, out: torch.Tensor = None, accumulate: bool = False) -> torch.Tensor:
    """fp32 [k, k] = x^T x (+ out) for a CUDA matrix x [n, k] (fp16 / bf16 / fp32)."""
    n, k = x.shape
    dev = x.device
    ld, step = x.stride()
    if not x.is_cuda or (k > 1 and step != 1):
        raise RuntimeError("expected a CUDA matrix with unit column stride")
    if out is None:
        out = torch.empty((k, k), dtype=torch.float32, device=dev)
        accumulate = False
        ldg = k
    else:
        ldg = _check_out(out, k, k, dev)
    lib = _lib.lib()
    with _lib.on_device(dev):
        stream = _lib.current_stream(dev)
        dt = _DTYPES[x.dtype]
        ws = _workspaces.take(dev, stream, lib.tb_gram_workspace_bytes(dt, n, k))
        _lib.check(lib.tb_gram(dev.index, stream, x.data_ptr(), dt, n, k, ld, out.data_ptr(), ldg, int(accumulate),
                               ws.data_ptr(), ws.numel()))
        _workspaces.give(dev, stream, ws)
    return out


def spd_inverse_(a: torch.Tensor, lambda_reg: float = 0.0, rescale: bool = True) -> torch.Tensor:
    """In place: a <- inv(a + lambda I) [/ mean |entry|] for a CUDA fp32 [k, k] matrix."""
    _launch_spd_inverse(a, lambda_reg, rescale)
    _lib.stream_status(a.device.index, _lib.current_stream(a.device))  # raises NotPositiveDefinite / DeviceTimeout
    return a


def _launch_spd_inverse(a: torch.Tensor, lambda_reg: float, rescale: bool) -> None:
    """``spd_inverse_`` without waiting for it: the caller checks ``device_status`` before it returns."""
    if a.dtype != torch.float32 or a.dim() != 2 or a.shape[0] != a.shape[1] or a.stride(1) != 1:
        raise RuntimeError("expected a square fp32 matrix with unit column stride")
    dev = a.device
    lib = _lib.lib()
    with _lib.on_device(dev):
        stream = _lib.current_stream(dev)
        ws = _workspaces.take(dev, stream, lib.tb_spd_inverse_workspace_bytes(a.shape[0]))
        _lib.check(lib.tb_spd_inverse(dev.index, stream, a.data_ptr(), a.shape[0], a.stride(0),
                                      float(lambda_reg), int(rescale), None, ws.data_ptr(), ws.numel()))
        _workspaces.give(dev, stream, ws)


def gemm_nt(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor = None, row_scale: torch.Tensor = None,
            alpha: float = 1.0, accumulate: bool = False, b_ready=None) -> torch.Tensor:
    """fp32 [M, N] = alpha * row_scale[:, None] * a @ b.T (+ out) for CUDA a [M, K], b [N, K].

    ``b_ready`` makes the current stream wait for ``b``, which an inverse on another stream is making; it is called when
    ``a`` has been laid out for the product, on half of the SMs."""
    if a.dtype != b.dtype:
        if b_ready is not None:
            b_ready()
            b_ready = None
        a, b = a.float(), b.float()
    (M, K), (N, Kb), dev = a.shape, b.shape, a.device
    (lda, step_a), (ldb, step_b) = a.stride(), b.stride()
    if Kb != K:
        raise RuntimeError("inner dimensions differ")
    if not a.is_cuda or b.device != dev or (K > 1 and (step_a != 1 or step_b != 1)):
        raise RuntimeError("expected CUDA matrices with unit column stride on one device")
    if out is None:
        out = torch.empty((M, N), dtype=torch.float32, device=dev)
        accumulate = False
        ldc = N
    else:
        ldc = _check_out(out, M, N, dev)
    if row_scale is not None:
        row_scale = row_scale.to(dev, torch.float32).reshape(-1).contiguous()
        if row_scale.numel() != M:
            raise RuntimeError("row_scale must have one entry per row of a")
    lib = _lib.lib()
    with _lib.on_device(dev):
        stream = _lib.current_stream(dev)
        dt = _DTYPES[a.dtype]
        ws = _workspaces.take(dev, stream, lib.tb_gemm_nt_workspace_bytes(dt, M, N, K))
        scale = row_scale.data_ptr() if row_scale is not None else None
        if b_ready is not None:
            _lib.check(lib.tb_gemm_nt_pack_beside(dev.index, stream, a.data_ptr(), lda, dt, M, N, K, ws.data_ptr(), ws.numel()))
            b_ready()
            _lib.check(lib.tb_gemm_nt_packed(dev.index, stream, b.data_ptr(), ldb, dt, M, N, K, out.data_ptr(), ldc,
                                             scale, float(alpha), int(accumulate), ws.data_ptr(), ws.numel()))
        else:
            _lib.check(lib.tb_gemm_nt(dev.index, stream, a.data_ptr(), lda, b.data_ptr(), ldb, dt, M, N, K,
                                      out.data_ptr(), ldc, scale, float(alpha), int(accumulate), ws.data_ptr(),
                                      ws.numel()))
        _workspaces.give(dev, stream, ws)
    return out


class B200ScoreComputer:
    """Drop-in for ``BasicScoreComputer`` on a B200."""

    def __init__(self, dtype: torch.dtype, device, CUDA_MAX_DIM_SIZE: int = 65_536,
                 logging_level=logging.INFO, lambda_reg: float = 0.0, process_group=None) -> None:
        self.dtype = dtype
        device = torch.device(device)
        if device.type != "cuda":
            raise ValueError("B200ScoreComputer only works on a CUDA device")
        if device.index is None:
            device = torch.device("cuda", torch.cuda.current_device())
        self.device = device
        self.CUDA_MAX_DIM_SIZE = CUDA_MAX_DIM_SIZE  # most rows moved to the GPU and multiplied at a time (_blocks)
        self.logger = logging.getLogger("ScoreComputer")
        self.logger.setLevel(logging_level)
        self.lambda_reg = lambda_reg
        self.process_group = process_group
        _lib.lib()

    # -- trak/score_computers.py:145-155
    def get_xtx(self, grads: torch.Tensor) -> torch.Tensor:
        self.proj_dim = grads.shape[1]
        accs = [None, None]   # one partial Gram per stream of the pair (blocks alternate between them)
        blocks = self._blocks(grads)
        with _lib.on_device(self.device), self._pair(len(blocks) > 1) as pair:
            for i, block in enumerate(blocks):
                with pair.stream(i):
                    blk = _as_device_matrix(block, self.device)
                    pair.uses(blk)
                    accs[i % 2] = gram(blk, out=accs[i % 2], accumulate=accs[i % 2] is not None)
        for a in accs:   # allocated on a side stream, used on the caller's from here on
            if a is not None:
                pair.uses(a)
        acc = accs[0]
        if acc is None:
            # a rank whose shard holds no rows still has to reach the all-reduce: it contributes zeros
            acc = torch.zeros(self.proj_dim, self.proj_dim, dtype=torch.float32, device=self.device)
        elif accs[1] is not None:
            acc.add_(accs[1])
        acc = reduce_gram(acc, self.process_group)
        _lib.stream_status(self.device.index, _lib.current_stream(self.device))
        return acc.to(self.dtype)

    # -- trak/score_computers.py:157-177
    def get_x_xtx_inv(self, grads: torch.Tensor, xtx: torch.Tensor) -> torch.Tensor:
        result = torch.empty(grads.shape[0], xtx.shape[1], dtype=self.dtype, device=self.device)
        start = 0
        blocks = self._blocks(grads)
        apart = len(blocks) > 1 or not grads.is_cuda or grads.numel() * grads.element_size() >= self.APART_BYTES
        with _lib.on_device(self.device), self._pair(apart) as pair:
            # the pair's streams do not wait for the inverse: the blocks are copied, converted and packed meanwhile
            inv = xtx.to(self.device, torch.float32, copy=True)
            _launch_spd_inverse(inv, self.lambda_reg, rescale=True)
            inv = inv.to(self.dtype)
            in_dtype = grads.dtype if grads.dtype in _DTYPES else torch.float32
            if in_dtype != inv.dtype:  # the narrower operand is promoted, never the inverse demoted
                inv = inv.to(torch.promote_types(in_dtype, inv.dtype))
            inverted = pair.mark()
            for i, block in enumerate(blocks):
                rows = slice(start, start + block.shape[0])
                start += block.shape[0]
                with pair.stream(i):
                    blk = _as_device_matrix(block, self.device).to(inv.dtype)
                    pair.uses(blk)
                    # (a third block comes behind a product that has waited for the inverse)
                    ready = (lambda: pair.after(inverted)) if apart and i < 2 else None
                    # the inverse is symmetric, so block @ inv == block @ inv.T
                    if result.dtype == torch.float32:
                        gemm_nt(blk, inv, out=result[rows], b_ready=ready)
                    else:
                        result[rows] = gemm_nt(blk, inv, b_ready=ready).to(self.dtype)
        _lib.stream_status(self.device.index, _lib.current_stream(self.device))  # raises NotPositiveDefinite / DeviceTimeout
        return result

    # A device matrix from this size on is packed on a stream of its own while the inverse, which leaves most of the device
    # idle, is computed: that hides 40 us and more (126 us at 50,000 x 2048 fp32) for about 20 us of host time.
    APART_BYTES = 128 << 20
    UPLOAD_BYTES = 96 << 20  # about so many bytes of a host matrix are uploaded at a time, under the work on the last

    def _blocks(self, t: torch.Tensor, rows: int = None):
        """The row blocks of ``t`` that are multiplied at a time; shorter ones for a matrix on the host."""
        rows = self.CUDA_MAX_DIM_SIZE if rows is None else rows
        if not t.is_cuda:
            rows = min(rows, max(8192, self.UPLOAD_BYTES // max(1, t.shape[1] * t.element_size()) // 256 * 256))
        return [b for b in torch.split(t, rows, dim=0) if b.shape[0]] if t.shape[0] > rows else [t] if t.shape[0] else []

    def _pair(self, wanted: bool):
        if not wanted:
            return OneStream(self.device)
        # one pair per thread and device, for all its computers: the workspaces are kept by stream
        pairs = _pairs.__dict__
        pair = pairs.get(self.device.index)
        if pair is None:
            pairs[self.device.index] = pair = StreamPair(self.device)
        return pair

    # -- trak/score_computers.py:179-189
    def get_scores(self, features: torch.Tensor, target_grads: torch.Tensor, accumulator: torch.Tensor,
                   row_scale: torch.Tensor = None) -> None:
        """``accumulator += features @ target_grads.T`` (times ``row_scale`` per train row when given).

        TRAKer keeps the accumulator on the host (trak/traker.py:632): the product then leaves the GPU in row
        blocks of at most ``HOST_STAGE_BYTES``, copied and added by several host threads while the GPU multiplies
        the next block, instead of one synchronous pageable copy per block."""
        _check_accumulator(features.shape[0], target_grads.shape[0], accumulator, row_scale)
        self._accumulate_products(features, _as_device_matrix(target_grads, self.device), accumulator, row_scale)

    def get_scores_from_grads(self, grads: torch.Tensor, xtx: torch.Tensor, target_grads: torch.Tensor,
                              accumulator: torch.Tensor, row_scale: torch.Tensor = None) -> None:
        """The same scores without materialising the features:
        ``accumulator += grads @ (inv @ target_grads.T)`` with ``inv`` the regularised, rescaled inverse of
        ``xtx`` exactly as ``get_x_xtx_inv`` forms it (trak/score_computers.py:157-168).  One product over
        the train rows instead of two: ``2 k^2 m`` flop for ``inv @ target_grads.T`` replace the ``2 n k^2``
        of the features.  For callers that do not need the features themselves (TRAKer stores them)."""
        _check_accumulator(grads.shape[0], target_grads.shape[0], accumulator, row_scale)
        inv = xtx.to(self.device, torch.float32, copy=True)
        spd_inverse_(inv, self.lambda_reg, rescale=True)   # raises before anything is added to the accumulator
        targets = _as_device_matrix(target_grads, self.device)
        solved = gemm_nt(targets.float(), inv)  # [m, k] = target_grads @ inv  (inv is symmetric)
        self._accumulate_products(grads, solved, accumulator, row_scale)

    def _accumulate_products(self, features, targets, accumulator, row_scale):
        m = targets.shape[0]
        on_host = accumulator.device.type == "cpu"
        exact = accumulator.shape[1] == m and not accumulator.requires_grad  # else torch's own += decides
        step = self.CUDA_MAX_DIM_SIZE
        if on_host:
            step = max(256, min(step, self.HOST_STAGE_BYTES // (4 * m) // 256 * 256))
            threaded = exact and accumulator.dtype == torch.float32 and accumulator.is_contiguous()
        pending = None

        def flush(item):
            rows, part, stream = item
            if threaded:
                mmap_io.device_to_host(accumulator[rows], part, stream, add=True)
                return
            with torch.cuda.stream(stream):
                accumulator[rows] += part.cpu().to(accumulator.dtype)

        start = 0
        blocks = self._blocks(features, step)
        with _lib.on_device(self.device), self._pair(len(blocks) > 1) as pair:
            for i, block in enumerate(blocks):
                rows = slice(start, start + block.shape[0])
                start += block.shape[0]
                with pair.stream(i):
                    blk = _as_device_matrix(block, self.device)
                    pair.uses(blk)
                    rs = None if row_scale is None else row_scale.reshape(-1)[rows]
                    into = accumulator[rows]
                    if exact and into.device == blk.device and into.dtype == torch.float32 and into.stride(1) == 1 \
                            and into.stride(0) >= m:
                        gemm_nt(blk, targets, out=into, row_scale=rs, accumulate=True)  # the epilogue's += is the same
                        continue
                    part = gemm_nt(blk, targets, row_scale=rs)
                    if not on_host:
                        if accumulator.device == part.device:
                            accumulator[rows] += part.to(accumulator.dtype)
                        else:
                            accumulator[rows] += part.to(accumulator.dtype).to(accumulator.device)
                        continue
                # the copy runs on this block's stream, under the GEMM of the next block on the other one
                if pending is not None:
                    flush(pending)
                pending = (rows, part, pair.current(i))
        if pending is not None:
            flush(pending)
        _lib.stream_status(self.device.index, _lib.current_stream(self.device))

    HOST_STAGE_BYTES = 128 << 20  # most bytes of scores that leave for a host accumulator at a time


def reduce_gram(local_gram: torch.Tensor, process_group=None) -> torch.Tensor:
    """Sums the per-rank Gram matrices when the train rows are sharded over a process group
    (the only exchange of the scoring path); a no-op for a single process."""
    import torch.distributed as dist
    if process_group is None:
        return local_gram
    if not (dist.is_available() and dist.is_initialized()):
        raise RuntimeError("process_group given but torch.distributed is not initialised")
    dist.all_reduce(local_gram, op=dist.ReduceOp.SUM, group=process_group)
    return local_gram


def shard_rows(n: int, rank: int, world: int):
    """Contiguous row range [lo, hi) of rank `rank` when n rows are split over `world` ranks."""
    base, rem = divmod(n, world)
    lo = rank * base + min(rank, rem)
    return lo, lo + base + (1 if rank < rem else 0)
