"""Many gradients side by side, each on two streams (steps and recompute), pass
after pass: every pass ends and gives the gradients of the instances run one
at a time. In a child process with a time limit, so that a stall fails the
test instead of stopping it."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

CHILD = """
import sys
import torch
from gbstencil import capi
from gbstencil.adjoint import Checkpointed, backward_batch, forward_batch
dtype = getattr(torch, sys.argv[1])
names, n, T, C = ["j2d5pt", "star2d2r", "box2d1r", "j2d9pt"] * 4, (400, 500), 32, 8
g = torch.Generator(device="cuda").manual_seed(61)
us = [torch.rand([x + 2 * capi.info(m)["rad"] for x in n], generator=g, device="cuda", dtype=dtype) for m in names]
want = [Checkpointed(m, u, T, C).backward(u, True) for m, u in zip(names, us)]
for _ in range(30):
    for _ in range(2):  # the second enqueued while the first runs
        runs = forward_batch(list(zip(names, us)), T, C)
        gu, gc = backward_batch(runs, us, True)
    done = torch.cuda.Event()
    done.record()
    done.synchronize()
    for (wu, wc), a, b in zip(want, gu, gc):
        assert torch.equal(wu, a) and torch.equal(wc, b)
"""


@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_sixteen_instances_pass_after_pass(dtype):
    env = dict(os.environ, PYTHONPATH=str(ROOT / "an5d-artifact_gb300"))
    r = subprocess.run([sys.executable, "-c", CHILD, dtype], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
