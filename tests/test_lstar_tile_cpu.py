"""The lower-star tile, compiled for the host, against the oracle (no GPU).

tests/lstar_tile_host.cpp drives msceer_gb300/csrc/lstar_tile.cuh over whole volumes with
arrays of exactly the kernel's sizes; its pairs and flags equal the oracle's.  Shapes around multiples of the
tiles' 32 x 4 x 4 (2D 32 x 16) vertices, ties, both zeros and infinities."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from msceer_gb300 import fields
from test_kernel_core_cpu import enc_map

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def tile(tmp_path_factory):
    out = tmp_path_factory.mktemp("tile") / "libtile.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out),
                    str(HERE / "lstar_tile_host.cpp")], check=True)
    lib = ctypes.CDLL(str(out))
    lib.tile_pairs.argtypes = [ctypes.c_int, ctypes.c_void_p] + [ctypes.c_int64] * 3 + [ctypes.c_void_p, ctypes.c_uint32]
    return lib


def make(kind, shape):
    if kind == "k3":
        return fields.power_law_field(shape, seed=5)
    rng = np.random.default_rng(7)
    if kind == "ties":
        return rng.integers(0, 4, size=shape[::-1]).astype(np.float32)
    return rng.choice(np.array([0.0, -0.0, np.inf, -np.inf, 1.0, -1e-42, 3e38, -3e38], dtype=np.float32), size=shape[::-1])


@pytest.mark.parametrize("kind", ["k3", "ties", "special"])
@pytest.mark.parametrize("shape", [(32, 4, 4), (33, 5, 5), (31, 3, 9), (70, 13, 6), (1, 7, 9), (2, 2, 2), (32, 16),
                                   (65, 17), (3, 40)], ids=lambda s: "x".join(map(str, s)))
def test_tile_equals_oracle(tile, oracle, kind, shape):
    f = np.ascontiguousarray(make(kind, shape))
    v = list(shape) + [1] * (3 - len(shape))
    g = np.zeros(int(np.prod([2 * n - 1 for n in shape])), dtype=np.uint8)
    tile.tile_pairs(len(shape), f.ctypes.data, *v, g.ctypes.data, enc_map(shape))
    want = oracle.grad(f)
    assert (g & 1).all()
    assert np.array_equal(g & 0x1F, want & 0x1F)  # assigned, flag and pairs; the closure sets the rest


@pytest.mark.parametrize("labels", ["random", "slab"])
@pytest.mark.parametrize("shape", [(32, 4, 4), (33, 5, 5), (70, 13, 6), (1, 7, 9), (2, 2, 2), (31, 3, 9)],
                         ids=lambda s: "x".join(map(str, s)))
def test_restricted_tile_equals_oracle(tile, oracle, shape, labels):
    f = np.ascontiguousarray(make("ties", shape))
    tile.tile_conform.argtypes = [ctypes.c_void_p] + [ctypes.c_int64] * 3 + [ctypes.c_void_p, ctypes.c_void_p,
                                                                             ctypes.c_uint32]
    tile.tile_conform.restype = ctypes.c_int64
    base = oracle.grad(f)
    rng = np.random.default_rng(3)
    if labels == "random":
        r = rng.integers(0, 4, size=base.size).astype(np.uint8)
    else:  # few restricted cells, so that some lower stars keep their pairs
        r = (rng.random(base.size) < 0.02).astype(np.uint8) * rng.integers(1, 4, size=base.size).astype(np.uint8)
    want = oracle.conform(f, r, base)
    g = base.copy().reshape(-1)
    assert tile.tile_conform(f.ctypes.data, *shape, r.ctypes.data, g.ctypes.data, enc_map(shape)) > 0
    assert np.array_equal(g & 0x1F, want.reshape(-1) & 0x1F)
