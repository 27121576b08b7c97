"""Extents that the entries refuse, and the largest they take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 262140  # along y


def test_image_rows(gpu, oracle):
    import torch
    from msceer_gb300 import _lib, lower_star_grad
    f = np.random.default_rng(1).standard_normal((ROWS + 1, 2)).astype(np.float32)
    assert np.array_equal(lower_star_grad(torch.from_numpy(f[:ROWS]).to(gpu)).cpu().numpy(), oracle.grad(f[:ROWS]))
    with pytest.raises(_lib.MscError):
        lower_star_grad(torch.from_numpy(f).to(gpu))


def test_network_rows(gpu):
    import torch
    from msceer_gb300 import _lib, triage
    feat = torch.zeros(16 * (ROWS + 1), dtype=torch.int16, device=gpu)
    w = triage.init_weights(0)
    _, _, logits = triage.forward(feat[:16 * ROWS], (1, ROWS, 1), w)
    assert torch.equal(logits, torch.zeros_like(logits))  # (no bias)
    with pytest.raises(_lib.MscError):
        triage.forward(feat, (1, ROWS + 1, 1), w)
