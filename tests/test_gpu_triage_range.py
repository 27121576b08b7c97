"""The triage network's gradients at the ends of the number range, against what the
definitions give: out = bf16(acc * (mask > 0)) with acc in FP32, and weight gradients that
are sums over the volume's own vertices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NW = 27 * 256


def _bits(x):
    """BF16 bits (int16 tensor) of values that BF16 holds."""
    import torch
    return torch.as_tensor(np.asarray(x, dtype=np.float32)).cuda().bfloat16().view(torch.int16)


@pytest.mark.parametrize("w_exp, masked, want", [(64, True, 0.0), (64, False, -np.inf), (65, True, np.nan),
                                                 (65, False, -np.inf)],
                         ids=["finite-masked", "finite", "infinite-masked", "infinite"])
def test_masked_gradient_that_rounds_to_infinity(gpu, w_exp, masked, want):
    """One vertex, one product: the logit gradient -(129/128) 2^63 times the weight (254/128)
    2^w_exp.  At 2^64 their product 1.9999 * 2^127 is finite in FP32 and infinite in BF16, at 2^65
    infinite in both; masked, the first is zero and the second NaN."""
    import torch
    from msceer_gb300 import triage
    w = torch.zeros(triage.PARAMS, device="cuda")
    w[2 * NW + 13 * 256: 2 * NW + 14 * 256].view(16, 16)[:, 0] = 254 / 128 * 2.0 ** w_exp
    a = _bits([0.0 if masked else 1.0] * 16)
    logits = torch.full((2, 1), -200.0, device="cuda")
    target = torch.tensor([[1], [0]], dtype=torch.uint8, device="cuda")
    _, g = triage.backward(_bits(np.zeros(16)), a, a, logits, target, (1, 1, 1), w, 2.0 * 129 / 128 * 2.0 ** 63)
    db2 = g[3 * NW + 16: 3 * NW + 32].cpu().numpy()
    assert np.array_equal(db2, np.full(16, want, dtype=np.float32), equal_nan=True), db2


@pytest.mark.parametrize("at", [(0, 3, 31), (0, 0, 0), (0, 3, 17)], ids=str)
def test_weight_gradient_of_an_infinite_feature(gpu, at):
    """A 32 x 4 x 1 volume with one infinite feature: the weight gradients that a vertex of the
    volume gives it are infinite, all others finite, whatever lies past the volume in its tile."""
    import torch
    from msceer_gb300 import triage
    shape = (1, 4, 32)
    rng = np.random.default_rng(4)
    feat = np.ones(shape + (16,), dtype=np.float32)
    feat[at + (0,)] = np.inf
    rows = _bits(np.stack([feat[..., :8], feat[..., 8:]], 2))
    w = torch.from_numpy(rng.uniform(0.5, 1.0, triage.PARAMS).astype(np.float32)).cuda()
    a = _bits(np.ones(16 * feat[..., 0].size))
    logits = torch.zeros((2, feat[..., 0].size), device="cuda")
    target = torch.zeros((2, feat[..., 0].size), dtype=torch.uint8, device="cuda")
    _, g = triage.backward(rows.reshape(-1), a, a, logits, target, shape, w, 1.0)
    g = g.cpu().numpy()
    dw1 = g[:NW].reshape(3, 3, 3, 16, 16)  # dz, dy, dx, cin, cout
    for dz in range(3):
        for dy in range(3):
            for dx in range(3):
                v = (at[0] - dz + 1, at[1] - dy + 1, at[2] - dx + 1)  # the vertex that sees the feature there
                inside = all(0 <= c < n for c, n in zip(v, shape))
                assert np.all(dw1[dz, dy, dx, 0] == np.inf) if inside else np.all(np.isfinite(dw1[dz, dy, dx, 0]))
    assert np.isfinite(dw1[..., 1:, :]).all() and np.isfinite(g[NW:]).all()
