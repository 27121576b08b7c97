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
