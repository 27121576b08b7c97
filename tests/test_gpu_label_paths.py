"""The FP32 streamlines' two stop tests -- the flags read with a voxel's corner gradients
(steps of less than half a voxel) and the nearest vertex's state in memory (any step) --
give the same labels, stages and iteration counts bit for bit where both apply, over thin
and odd volumes (every voxel next to the boundary), step bounds up to the rule's limit and
the iteration limit's edges.  The switch is read once per process, so each form runs in a
child process."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

CHILD = r"""
import hashlib, json, sys
sys.path.insert(0, sys.argv[1])
import torch
from msceer_gb300 import fields, integrated_labels, lower_star_grad
out = []
for shape in [(2, 2, 2), (3, 5, 40), (4, 33, 9), (37, 29, 31), (64, 40, 48)]:
    for kind in ("gauss", "k3"):
        f = fields.gaussian_sum(shape, 9, seed=3) if kind == "gauss" else fields.power_law_field(shape, seed=8)
        f = torch.from_numpy(f).cuda()
        g = lower_star_grad(f)
        for kw in ({}, {"max_step": 0.45, "error_threshold": 1e-3}, {"max_step": 0.03}, {"iteration_limit": 16},
                   {"iteration_limit": 65, "precision": 2}, {"max_step": 0.5}):
            r = integrated_labels(f, g, stages=True, **kw)
            out.append([shape, kind, str(kw), {k: v if k == "stats" else hashlib.sha256(v.cpu().numpy().tobytes()).hexdigest()
                                               for k, v in r.items()}])
print(json.dumps(out))
"""


def _run(extra):
    p = subprocess.run([sys.executable, "-c", CHILD, str(ROOT)], env=dict(os.environ, **extra), capture_output=True,
                       text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


def test_stop_tests_agree(gpu):
    a, b = _run({}), _run({"MSC_STOP_TEST": "memory"})
    assert len(a) == len(b) == 60
    for x, y in zip(a, b):
        assert x == y, x[:3]
