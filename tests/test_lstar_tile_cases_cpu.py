"""The lower-star tile that the kernels run (msceer_gb300/csrc/lstar_tile.cuh), compiled for
the host, on the golden fields, random fields and conforming labels that the per-vertex form
is checked on: bytes with the ascending-manifold roots as the kernel writes them, and after the
oracle's closure the oracle's .grad (no GPU)."""
import ctypes

import numpy as np
import pytest

import oracle_lib
from msceer_gb300 import fields
from test_kernel_core_cpu import enc_map
from test_lstar_tile_cpu import tile  # noqa: F401


def roots(grad, dims):
    """The closure's roots in place of the ldir bits: critical 1-, 2-, 3-cells 2, 1, 0, the rest 3."""
    d = [2 * v - 1 for v in dims]
    ids = np.arange(grad.size)
    dim = sum((c & 1) for c in [ids % d[0], (ids // d[0]) % d[1]] + ([ids // (d[0] * d[1])] if len(dims) == 3 else []))
    crit = ((grad >> 2) & 7) == 7
    return np.where(crit & (dim > 0), 3 - dim, 3).astype(np.uint8)


def check(tile, oracle, f):  # noqa: F811
    f = np.ascontiguousarray(f, dtype=np.float32)
    dims = f.shape[::-1]
    got = np.zeros(int(np.prod([2 * v - 1 for v in dims])), dtype=np.uint8)
    tile.tile_pairs(len(dims), f.ctypes.data, *(list(dims) + [1] * (3 - len(dims))), got.ctypes.data, enc_map(dims))
    want = oracle.grad(f)
    assert np.array_equal(got & 0x1F, want & 0x1F), oracle_lib.describe_mismatch(got & 0x1F, want & 0x1F, dims)
    assert np.array_equal(got >> 5, roots(want, dims))
    assert np.array_equal(oracle.ldir(got, dims), want)


@pytest.mark.parametrize("case", oracle_lib.load_golden_small(), ids=lambda c: c[0])
def test_tile_golden(tile, oracle, case):  # noqa: F811
    check(tile, oracle, case[1])


SHAPES = [(31, 17, 9), (40, 37, 1), (1, 20, 23), (48, 48, 48), (300, 211), (1, 40), (40, 1)]


@pytest.mark.parametrize("shape, kind", [(s, k) for s in SHAPES for k in ("k3", "quant3", "gauss")
                                         if k != "gauss" or len(s) == 3], ids=str)
def test_tile_random(tile, oracle, shape, kind):  # noqa: F811
    if kind == "gauss":
        f = fields.gaussian_sum(shape, 8, seed=3)
    else:
        f = fields.power_law_field(shape, seed=5)
        if kind == "quant3":
            f = fields.quantized(f, 3)
    check(tile, oracle, f)


@pytest.mark.parametrize("shape", [(40, 36, 32), (31, 17, 9), (33, 2, 20)], ids=lambda s: "x".join(map(str, s)))
def test_tile_conform(tile, oracle, shape):  # noqa: F811
    """The re-pairing from the restriction labels of the oracle's own final labels."""
    f = np.ascontiguousarray(fields.gaussian_sum(shape, 8, seed=5))
    gt = 1e-6 * float(np.abs(f).max())
    base = oracle.grad(f)
    lab = oracle.labels(f, base, 1e-4, gt, 4000, 0.25, 0.0)
    restrict = oracle.boundary_labels(f, lab["asc"], lab["dsc"])
    want = oracle.conform(f, restrict, base)
    dims = f.shape[::-1]
    got = base.copy()
    tile.tile_conform.argtypes = [ctypes.c_void_p] + [ctypes.c_int64] * 3 + [ctypes.c_void_p, ctypes.c_void_p,
                                                                             ctypes.c_uint32]
    tile.tile_conform.restype = ctypes.c_int64
    assert tile.tile_conform(f.ctypes.data, *dims, restrict.ctypes.data, got.ctypes.data, enc_map(dims)) > 0
    got = (got & 0x1F) | (roots(got, dims) << 5)
    assert np.array_equal(oracle.ldir(got, dims), want), oracle_lib.describe_mismatch(oracle.ldir(got, dims), want, dims)
