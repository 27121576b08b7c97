"""The block-shared frontier walks (the .grad's ascending-manifold closure across tiles, the
labels' certain terminal regions) on fields whose chains are long: one basin over the
whole volume, a ramp, a plateau of equal values, a smooth sum of Gaussians, and a rough
field beside them.  Bytes and labels equal the oracle's (no tolerance)."""
import numpy as np
import pytest

from msceer_gb300 import fields

pytestmark = pytest.mark.gpu


def one_basin(shape):
    z, y, x = np.meshgrid(*[np.arange(n, dtype=np.float64) for n in shape[::-1]], indexing="ij")
    c = [0.4 * n for n in shape]
    return ((x - c[0]) ** 2 + 1.3 * (y - c[1]) ** 2 + 0.7 * (z - c[2]) ** 2).astype(np.float32)


def ramp(shape):
    z, y, x = np.meshgrid(*[np.arange(n, dtype=np.float64) for n in shape[::-1]], indexing="ij")
    return (x + 1.7 * y + 0.3 * z).astype(np.float32)


FIELDS = {
    "basin": one_basin,
    "ramp": ramp,
    "plateau": lambda s: np.zeros(s[::-1], dtype=np.float32),
    "smooth": lambda s: fields.gaussian_sum(s, 6, seed=2, noise=1e-6),
    "k3": lambda s: fields.power_law_field(s, seed=9),
}


@pytest.mark.parametrize("name", list(FIELDS))
@pytest.mark.parametrize("shape", [(2, 2, 2), (31, 17, 5), (61, 40, 70)], ids=lambda s: "x".join(map(str, s)))
def test_closure_walk_equals_oracle(gpu, oracle, name, shape):
    import torch
    from msceer_gb300 import lower_star_grad
    f = FIELDS[name](shape)
    assert np.array_equal(lower_star_grad(torch.from_numpy(f).to(gpu)).cpu().numpy(), oracle.grad(f))


def test_closure_walk_2d(gpu, oracle):
    import torch
    from msceer_gb300 import lower_star_grad
    f = fields.gaussian_sum((300, 611), 9, seed=4, noise=1e-6)
    assert np.array_equal(lower_star_grad(torch.from_numpy(f).to(gpu)).cpu().numpy(), oracle.grad(f))


@pytest.mark.parametrize("name", list(FIELDS))
@pytest.mark.parametrize("shape", [(2, 2, 2), (9, 21, 6), (44, 36, 40)], ids=lambda s: "x".join(map(str, s)))
def test_terminal_walk_equals_oracle(gpu, oracle, name, shape):
    import torch
    from msceer_gb300 import integrated_labels
    f = FIELDS[name](shape)
    g = oracle.grad(f)
    # few iterations: the terminal regions come before any streamline
    got = integrated_labels(torch.from_numpy(f).to(gpu), torch.from_numpy(g).to(gpu), 1e-4, 1e-6, 20, 0.25, 0.0, stages=True)
    want = oracle.labels(f, g, 1e-4, 1e-6, 20, 0.25, 0.0)
    for k in ("asc_terminal", "dsc_terminal"):
        assert np.array_equal(got[k].cpu().numpy(), want[k].reshape(-1)), k


# cells per axis 2n - 1 around multiples of the tiles' 28 owned cells (3D, and 2D along x)
# and 124 (2D along y); X = 1 gives the remapped pair codes
@pytest.mark.parametrize("shape", [(14, 15, 16), (15, 29, 14), (43, 14, 30), (1, 31, 29), (28, 62), (15, 63), (30, 125)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("offset", [0, 1, 7, 14])
def test_tile_edges_and_byte_alignment(gpu, oracle, shape, offset):
    """The bit-row tiles at their edges, in a .grad buffer at any byte offset; the bytes
    around the buffer stay as they were."""
    import torch
    from msceer_gb300 import lower_star_grad
    f = fields.gaussian_sum(shape, 5, seed=6, noise=1e-2)
    want = oracle.grad(f)
    buf = torch.full((want.size + 32,), 0xA5, dtype=torch.uint8, device=gpu)
    out = buf[offset:offset + want.size]
    lower_star_grad(torch.from_numpy(f).to(gpu), out)
    assert np.array_equal(out.cpu().numpy(), want)
    assert bool((buf[:offset] == 0xA5).all()) and bool((buf[offset + want.size:] == 0xA5).all())


@pytest.mark.parametrize("shape", [(33, 9, 10), (67, 40)], ids=lambda s: "x".join(map(str, s)))
def test_zeros_and_infinities(gpu, oracle, shape):
    """Both zeros, infinities, a denormal and the largest values, many of them equal: the
    order is by value, then index."""
    import torch
    from msceer_gb300 import lower_star_grad
    rng = np.random.default_rng(7)
    vals = np.array([0.0, -0.0, np.inf, -np.inf, 1.0, -1e-42, 3e38, -3e38], dtype=np.float32)
    f = rng.choice(vals, size=shape[::-1])
    assert np.array_equal(lower_star_grad(torch.from_numpy(f).to(gpu)).cpu().numpy(), oracle.grad(f))
