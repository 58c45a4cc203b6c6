"""The work a user of this library has it do, as timed cases through the public classes.

Three kinds of work make up a TRAK run, and every case is one of them:

``project``    per-sample gradients onto the JL matrix: ``CudaProjector.project`` (a gradient matrix or the dict of
               per-parameter tensors, matrix regenerated or stored) and ``ChunkedCudaProjector.project``
``score``      ``B200ScoreComputer``: Gram, regularised inverse and features, scores (or the scores without the
               features), on device tensors or on host tensors with a host accumulator as ``TRAKer`` calls it
``finalize``   ``ScoreFinalizer`` over the host stores of several checkpoints

Values are synthetic: gradients N(0, 1e-2), projected gradients N(0, 1/k), out-to-loss weights uniform in (0, 1).
"""
import math
import random

import numpy as np
import torch

from trak_b200.finalize import ScoreFinalizer
from trak_b200.projectors import CudaProjector, ProjectionType, make_chunked_projector
from trak_b200.score_computers import B200ScoreComputer

_DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
_BYTES = {"f16": 2, "bf16": 2, "f32": 4}
_PROJ_SEED = 17
_LAMBDA = 1e-3


# ---- parameter shapes ----------------------------------------------------------------------------------------
def _resnet18_widths(classes=10):
    """The 62 parameters of a CIFAR ResNet-18 (3x3 stem, no max-pool), in order: 11,173,962 features."""
    widths = [64 * 3 * 9, 64, 64]
    cin = 64
    for cout in (64, 128, 256, 512):
        for block in range(2):
            widths += [cout * cin * 9, cout, cout, cout * cout * 9, cout, cout]
            if block == 0 and cin != cout:
                widths += [cout * cin, cout, cout]
            cin = cout
    return widths + [classes * 512, classes]


def _gpt2_small_widths():
    """The 148 parameters of GPT-2-small, in order: 124,439,808 features."""
    d = 768
    layer = [d, d, 3 * d * d, 3 * d, d * d, d, d, d, 4 * d * d, 4 * d, 4 * d * d, d]
    return [50257 * d, 1024 * d] + 12 * layer + [d, d]


def _split_widths(features, tensors, seed):
    """`tensors` parameter widths that add up to `features`, spread over several orders of magnitude."""
    rng = random.Random(seed)
    weights = [math.exp(rng.uniform(0.0, 8.0)) for _ in range(tensors)]
    scale = (features - tensors) / sum(weights)
    widths = [1 + int(w * scale) for w in weights]
    widths[-1] += features - sum(widths)
    return widths


def _widths(case):
    layout = case["layout"]
    if layout == "resnet18":
        return _resnet18_widths()
    if layout == "gpt2_small":
        return _gpt2_small_widths()
    return _split_widths(case["features"], case["tensors"], case["split_seed"])


# ---- the cases -----------------------------------------------------------------------------------------------
def _project(name, rows, features, proj_dim, proj_type, dtype, layout="matrix", **more):
    case = {"name": name, "kind": "project", "rows": rows, "features": features, "proj_dim": proj_dim,
            "proj_type": proj_type, "dtype": dtype, "layout": layout, "stored": False, "chunk": 0}
    return dict(case, **more)


def _score(name, rows, proj_dim, targets, dtype, where="device", **more):
    case = {"name": name, "kind": "score", "rows": rows, "proj_dim": proj_dim, "targets": targets, "dtype": dtype,
            "where": where, "weights": False, "features_kept": True}
    return dict(case, **more)


def _finalize(name, rows, proj_dim, targets, checkpoints, dtype, out_dtype):
    return {"name": name, "kind": "finalize", "rows": rows, "proj_dim": proj_dim, "targets": targets,
            "checkpoints": checkpoints, "dtype": dtype, "out_dtype": out_dtype}


def listed():
    return [
        # a linear probe or a small classifier head, one small batch: the call itself is what costs
        _project("project_smallest", 16, 20_011, 512, "rademacher", "f32"),
        # a small network with the batch of the widest reference kernel
        _project("project_rademacher_32", 32, 1_048_576, 2048, "rademacher", "f32"),
        # featurizing CIFAR with a ResNet-18: what vmap(grad) returns goes to the projector as it is
        _project("project_rademacher_dict", 128, 11_173_962, 2048, "rademacher", "f32", layout="resnet18"),
        # a language model whose gradient is projected in parameter chunks, few rows at a time
        _project("project_chunked_bf16", 16, 124_439_808, 8192, "rademacher", "bf16", layout="gpt2_small",
                 chunk=40_000_000),
        # the headline: Gaussian matrix, half-precision gradients of a ResNet-18
        _project("project_normal_128", 128, 11_173_962, 4096, "normal", "f16"),
        # a large Gaussian batch of odd sizes in bf16
        _project("project_normal_ragged", 387, 1_000_003, 1024, "normal", "bf16"),
        # many batches of one checkpoint against a Gaussian matrix kept in device memory
        _project("project_normal_stored", 256, 2_097_169, 4096, "normal", "f16", stored=True),
        # scoring a small data set: a chain of short launches
        _score("score_small", 1_000, 512, 100, "f32"),
        # CIFAR-10 with the default projection size, on the device, with out-to-loss weights
        _score("score_ordinary", 50_000, 2048, 1_000, "f32", weights=True),
        # the same from half-precision host stores into a host accumulator, as TRAKer drives it
        _score("score_host_f16", 50_000, 2048, 1_003, "f16", where="host"),
        # one block of a million-example job
        _score("score_large", 65_613, 8192, 2_500, "f32"),
        # scores of three checkpoints, averaged and weighted, into the host score store
        _finalize("finalize_3_checkpoints", 50_000, 2048, 1_000, 3, "f16", "f16"),
    ]


# Bounds of the drawn cases; none costs more than the largest listed ones.
_MAX_MATRIX = 4.5e10        # matrix entries generated in one projection
_MAX_FLOPS = 1.2e13
_MAX_GRAD_BYTES = 5.5e9
_MAX_STORED = 8.0e9         # entries of a stored matrix
_MAX_HOST_BYTES = 6.0e8


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_project(rng):
    stored = rng.random() < 0.15
    rows = _log(rng, 1, 512)
    proj_dim = rng.choice([512, 1024, 1536, 2048, 4096, 8192])
    dtype = rng.choice(["f16", "bf16", "f32"])
    most = min((_MAX_STORED if stored else _MAX_MATRIX) / proj_dim, _MAX_FLOPS / (2.0 * rows * proj_dim),
               _MAX_GRAD_BYTES / (rows * _BYTES[dtype]))
    features = _log(rng, 7_690, most)
    more = {"stored": stored}
    if rng.random() < 0.4 and not stored:
        tensors = _log(rng, 4, 160)
        more.update(layout="split", tensors=tensors, split_seed=rng.randrange(1 << 20))
        if rng.random() < 0.3 and features > 200_000:
            widest = max(_split_widths(features, tensors, more["split_seed"]))
            more["chunk"] = widest + 1 + _log(rng, features // 8, features)
    proj_type = "normal" if stored else rng.choice(["rademacher", "rademacher", "normal"])
    if more.get("chunk"):
        proj_type = "rademacher"   # what the chunked projector is made of
    return _project("", rows, features, proj_dim, proj_type, dtype, **more)


def _draw_score(rng):
    proj_dim = rng.choice([_log(rng, 128, 8192) // 128 * 128, rng.choice([512, 1024, 2048, 4096]), _log(rng, 100, 3000)])
    where = rng.choice(["device", "device", "host"])
    dtype = rng.choice(["f32", "f16", "f32"])
    targets = _log(rng, 10, 10_000)
    most = _MAX_FLOPS / (3.0 * proj_dim ** 2 + 2.0 * targets * proj_dim)
    if where == "host":
        most = min(most, _MAX_HOST_BYTES / (proj_dim * _BYTES[dtype] + 4 * targets))
    rows = _log(rng, 3 * proj_dim, max(3 * proj_dim + 1, min(80_000, most)))
    if where == "host":   # the least rows may be many targets wide
        targets = min(targets, max(10, int(_MAX_HOST_BYTES / (4 * rows))))
    return _score("", rows, proj_dim, targets, dtype, where=where, weights=rng.random() < 0.5,
                  features_kept=rng.random() < 0.75)


def _draw_finalize(rng):
    proj_dim = rng.choice([512, 1024, 2048, 4096])
    dtype, out_dtype = rng.choice(["f16", "f32"]), rng.choice(["f16", "f32"])
    checkpoints, targets = rng.randint(1, 5), _log(rng, 10, 5_000)
    most = _MAX_HOST_BYTES / (checkpoints * proj_dim * _BYTES[dtype] + targets * _BYTES[out_dtype])
    return _finalize("", _log(rng, 1_000, min(80_000, most)), proj_dim, targets, checkpoints, dtype, out_dtype)


def draw(rng):
    pick = rng.random()
    case = _draw_project(rng) if pick < 0.55 else _draw_score(rng) if pick < 0.9 else _draw_finalize(rng)
    del case["name"]
    return case


# ---- inputs and runs -----------------------------------------------------------------------------------------
def _randn(gen, shape, dtype, scale):
    """N(0, scale) on the GPU, made in slices so that no fp32 copy of a large 16-bit tensor is held."""
    out = torch.empty(shape, dtype=dtype, device="cuda")
    flat = out.view(-1)
    step = 1 << 28
    for i in range(0, flat.numel(), step):
        part = flat[i:i + step]
        part.normal_(0.0, scale, generator=gen)
    return out


def _prepare_project(case, gen):
    dtype, rows = _DTYPES[case["dtype"]], case["rows"]
    if case["layout"] == "matrix":
        grads = _randn(gen, (rows, case["features"]), dtype, 1e-2)
        widths = [case["features"]]
    else:
        widths = _widths(case)
        grads = {f"p{i}": _randn(gen, (rows, w), dtype, 1e-2) for i, w in enumerate(widths)}
    if case["chunk"]:
        projector = make_chunked_projector(widths, case["proj_dim"], 0, rows, "cuda", dtype,
                                           max_chunk_size=case["chunk"])
    else:
        projector = CudaProjector(sum(widths), case["proj_dim"], _PROJ_SEED, ProjectionType(case["proj_type"]),
                                  "cuda", store_matrix=case["stored"])
    if case["stored"]:
        # the matrix is made by the first batch of a checkpoint and kept for the others
        projector.project(grads[:1], 0)
    return {"kind": "project", "projector": projector, "grads": grads}


def _prepare_score(case, gen):
    dtype, n, k, m = _DTYPES[case["dtype"]], case["rows"], case["proj_dim"], case["targets"]
    x = _randn(gen, (n, k), dtype, k ** -0.5)
    t = _randn(gen, (m, k), dtype, k ** -0.5)
    w = torch.rand(n, device="cuda", generator=gen) if case["weights"] else None
    acc = torch.zeros(n, m, device="cuda")
    if case["where"] == "host":
        x, t, acc = x.cpu(), t.cpu(), acc.cpu()
    return {"kind": "score", "computer": B200ScoreComputer(dtype, "cuda", lambda_reg=_LAMBDA), "x": x, "targets": t,
            "weights": w, "accumulator": acc, "features_kept": case["features_kept"]}


def _prepare_finalize(case, gen):
    dtype, n, k, m = _DTYPES[case["dtype"]], case["rows"], case["proj_dim"], case["targets"]
    feats = [_randn(gen, (n, k), dtype, 1.0).cpu().numpy() for _ in range(case["checkpoints"])]
    targets = [_randn(gen, (m, k), dtype, k ** -0.5).cpu().numpy() for _ in range(case["checkpoints"])]
    weights = [torch.rand(n, 1, device="cuda", generator=gen).to(dtype).cpu().numpy()
               for _ in range(case["checkpoints"])]
    scores = np.zeros((n, m), dtype=np.float16 if case["out_dtype"] == "f16" else np.float32)
    return {"kind": "finalize", "finalizer": ScoreFinalizer(feats, targets, weights, "cuda"), "scores": scores}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    make = {"project": _prepare_project, "score": _prepare_score, "finalize": _prepare_finalize}[case["kind"]]
    return make(case, gen)


def run(state):
    if state["kind"] == "project":
        return state["projector"].project(state["grads"], model_id=0)
    if state["kind"] == "finalize":
        return state["finalizer"].run(state["scores"])
    computer, acc = state["computer"], state["accumulator"]
    acc.zero_()
    xtx = computer.get_xtx(state["x"])
    if not state["features_kept"]:
        computer.get_scores_from_grads(state["x"], xtx, state["targets"], acc, row_scale=state["weights"])
        return {"xtx": xtx, "scores": acc}
    features = computer.get_x_xtx_inv(state["x"], xtx)
    computer.get_scores(features, state["targets"], acc, row_scale=state["weights"])
    return {"xtx": xtx, "features": features, "scores": acc}


# ---- what a pass cannot do without, and how exact it is --------------------------------------------------------
def work(case):
    e = _BYTES[case["dtype"]]
    n, k = case["rows"], case["proj_dim"]
    if case["kind"] == "project":
        f = case["features"]
        matrix = 2.0 * f * k if case["stored"] else 0.0
        out = n * k * (e if case["chunk"] else 4)
        return {"bytes": float(n * f * e + out) + matrix, "flops": 2.0 * n * f * k}
    m = case["targets"]
    if case["kind"] == "finalize":
        c, eo = case["checkpoints"], _BYTES[case["out_dtype"]]
        return {"bytes": float(c * (n + m) * k * e + c * n * e + n * m * eo), "flops": 2.0 * c * n * m * k}
    flops = float(n) * k * (k + 1) + float(k) ** 3 + 2.0 * n * m * k
    nbytes = float((n + m) * k * e + k * k * e + n * m * 4)
    if case["features_kept"]:
        return {"bytes": nbytes + n * k * e, "flops": flops + 2.0 * n * k * k}
    return {"bytes": nbytes, "flops": flops + 2.0 * m * k * k}


def tolerance(case):
    if case["kind"] == "project":
        # 16-bit products summed in 32 bits over up to 1e8 features; the chunked projector returns the gradients' dtype
        if case["chunk"] and case["dtype"] != "f32":
            return {"rel": 4e-3 if case["dtype"] == "bf16" else 5e-4}
        return {"rel": 1e-4}
    if case["kind"] == "finalize":
        return {"rel": 5e-4 if case["out_dtype"] == "f16" else 1e-5}
    # Gram, inverse and features are each rounded to the computer's dtype
    return {"rel": 3e-3 if case["dtype"] == "f16" else 1e-4}
