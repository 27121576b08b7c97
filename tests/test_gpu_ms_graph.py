"""The Morse-Smale complex graph of a device .grad (msc_ms_graph_3d) against the
reference's MorseSmaleComplexBasic::ComputeFromGrad: the golden fixture holds the
reference's own nodes and arcs (SHA-256 per array, tests/golden/make_ms_graph_golden.py),
larger fields are checked against the oracle, which equals the reference on every
golden case (tests/test_oracle.py)."""
import ctypes
import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

from msceer_gb300 import fields

pytestmark = pytest.mark.gpu

CASES = json.loads((Path(__file__).resolve().parent / "golden" / "ms_graph.json").read_text())


def _digests(graph):
    return {k: hashlib.sha256(np.ascontiguousarray(v.cpu().numpy()).tobytes()).hexdigest() for k, v in graph.items()}


def _device_graph(gpu, f, build):
    import torch
    from msceer_gb300 import lower_star_grad, ms_graph
    t = torch.from_numpy(np.ascontiguousarray(f)).to(gpu)
    g = lower_star_grad(t)
    return g, ms_graph(g, t, build)


@pytest.mark.parametrize("key", sorted(CASES))
def test_ms_graph_equals_reference_golden(gpu, key):
    spec = CASES[key]
    f = eval("fields." + spec["generator"], {"fields": fields}).astype(np.float32)
    g, got = _device_graph(gpu, f, spec["build_arcs"])
    assert hashlib.sha256(g.cpu().numpy().tobytes()).hexdigest() == spec["grad_sha256"]
    assert (got["node_cell"].numel(), got["arc_lower"].numel()) == (spec["nodes"], spec["arcs"])
    d = _digests(got)
    same_f = hashlib.sha256(f.tobytes()).hexdigest() == spec["f_sha256"]
    # the node values (and persistences) are f's own floats: compared where this host
    # regenerated the reference's exact input (the FFT fields can differ in their last
    # bits between hosts; test_ms_graph_128_cubed_vs_oracle covers the values there)
    keys = spec["sha256"] if same_f else [k for k in spec["sha256"] if k not in ("node_value", "arc_persistence")]
    assert {k: d[k] for k in keys} == {k: spec["sha256"][k] for k in keys}


@pytest.mark.parametrize("build", [(1, 0, 1), (1, 1, 1)])
def test_ms_graph_128_cubed_vs_oracle(gpu, oracle, build):
    f = fields.power_law_field((128, 128, 128), seed=9)
    g, got = _device_graph(gpu, f, build)
    want = oracle.ms_graph(f, g.cpu().numpy(), build)
    for k, v in want.items():
        assert np.array_equal(got[k].cpu().numpy(), v), k


def test_ms_graph_counts_only_then_fill(gpu):
    """Capacities 0 return the counts and write nothing; a second call fills."""
    import torch
    from msceer_gb300 import _lib, lower_star_grad, num_cells
    f = fields.gaussian_sum((24, 20, 16), 6, seed=2)
    t = torch.from_numpy(f).to(gpu)
    g = lower_star_grad(t)
    lib = _lib.load()
    dims = _lib.dims_arg(f.shape[::-1])
    counts = (ctypes.c_int64 * 2)(-1, -1)
    build = (ctypes.c_int * 3)(1, 1, 1)
    s = ctypes.c_void_p(torch.cuda.current_stream(gpu).cuda_stream)
    p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    rc = lib.msc_ms_graph_3d(p(g), p(t), dims, build, 0, None, None, None, None, 0, None, None, None, counts, s)
    assert rc == 0 and counts[0] > 0 and counts[1] > 0
    nn, na = counts[0], counts[1]
    cell = torch.full((nn,), -7, dtype=torch.int64, device=gpu)
    val = torch.empty(nn, dtype=torch.float32, device=gpu)
    dim = torch.empty(nn, dtype=torch.uint8, device=gpu)
    bnd = torch.empty(nn, dtype=torch.uint8, device=gpu)
    lo = torch.full((na,), -7, dtype=torch.int32, device=gpu)
    up = torch.empty(na, dtype=torch.int32, device=gpu)
    # too small an arc capacity: nodes written, arcs left alone
    rc = lib.msc_ms_graph_3d(p(g), p(t), dims, build, nn, p(cell), p(val), p(dim), p(bnd), na - 1, p(lo), p(up), None,
                             counts, s)
    assert rc == 0 and (counts[0], counts[1]) == (nn, na)
    assert bool((cell >= 0).all()) and bool((lo == -7).all())
    rc = lib.msc_ms_graph_3d(p(g), p(t), dims, build, nn, p(cell), p(val), p(dim), p(bnd), na, p(lo), p(up), None,
                             counts, s)
    assert rc == 0
    assert bool((lo >= 0).all()) and bool((lo < nn).all()) and bool((up < nn).all())
    # every arc joins a node to one a dimension lower
    assert bool((dim[lo.long()].int() + 1 == dim[up.long()].int()).all())
    assert num_cells(f.shape[::-1]) == g.numel()


@pytest.mark.parametrize("noise", [0.0, 8.0, 60.0])
@pytest.mark.parametrize("shape", [(2, 2, 2), (17, 9, 16), (1, 40, 33), (40, 33, 30)],
                         ids=lambda s: "x".join(map(str, s)))
def test_ms_graph_one_peak_vs_oracle(gpu, oracle, shape, noise):
    """Cell counts around the words and blocks of the node index, and one peak under noise:
    nodes with far more arcs than a tracing thread keeps (up to 1,647 at 40x33x30), and more
    arcs than the room for kept ones."""
    z, y, x = np.meshgrid(*[np.arange(n, dtype=np.float64) for n in shape[::-1]], indexing="ij")
    f = -((x - 0.5 * shape[0]) ** 2 + (y - 0.5 * shape[1]) ** 2 + (z - 0.5 * shape[2]) ** 2).astype(np.float32)
    f += np.random.default_rng(3).uniform(-noise, noise, size=f.shape).astype(np.float32)
    g, got = _device_graph(gpu, f, (1, 1, 1))
    want = oracle.ms_graph(f, g.cpu().numpy(), (1, 1, 1))
    for k, v in want.items():
        assert np.array_equal(got[k].cpu().numpy(), v), k


def test_ms_graph_allocator(gpu):
    """The one-call form: each array asked for once with its final length, the result that of
    the sized call, an allocator that fails ends the call."""
    import torch
    from msceer_gb300 import _lib, lower_star_grad, ms_graph
    f = torch.from_numpy(fields.power_law_field((30, 27, 25), seed=2)).to(gpu)
    g = lower_star_grad(f)
    want = ms_graph(g, f, (1, 1, 1))
    lib, p = _lib.load(), lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    s = ctypes.c_void_p(torch.cuda.current_stream(gpu).cuda_stream)
    counts, build, asked = (ctypes.c_int64 * 2)(), (ctypes.c_int * 3)(1, 1, 1), []
    fail = _lib.GRAPH_ALLOC(lambda ctx, array, count: asked.append((array, count)))
    assert lib.msc_ms_graph_alloc_3d(p(g), p(f), _lib.dims_arg((30, 27, 25)), build, fail, None, counts, s) == -4
    assert asked == [(a, want["node_cell"].numel()) for a in range(4)]
    assert lib.msc_ms_graph_alloc_3d(p(g), p(f), _lib.dims_arg((30, 27, 25)), build, _lib.GRAPH_ALLOC(), None, counts, s) == -2
    nn, na = want["node_cell"].numel(), want["arc_lower"].numel()
    got = {k: torch.empty_like(v) for k, v in want.items()}
    rc = lib.msc_ms_graph_3d(p(g), p(f), _lib.dims_arg((30, 27, 25)), build, nn, *[p(got[k]) for k in list(got)[:4]], na,
                             *[p(got[k]) for k in list(got)[4:]], counts, s)
    assert rc == 0 and (counts[0], counts[1]) == (nn, na)
    for k in want:
        assert torch.equal(got[k], want[k]), k
