"""Coefficient gradients keep their bits whatever the process ran before: the
binomial schedule (single steps) in a fresh process, then the full stash
(launches of two), then both again; and a first chunk of one step."""
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
from gbstencil.adjoint import Checkpointed
name, n, T, C = sys.argv[1], int(sys.argv[2]), 9, 4
r = capi.info(name)["rad"]
g = torch.Generator(device="cuda").manual_seed(41)
u0 = torch.rand([n + 2 * r] * 2, generator=g, device="cuda")
w = torch.rand([n + 2 * r] * 2, generator=g, device="cuda") - 0.5
out = []
for slots in [int(x) for x in sys.argv[3].split(",")]:
    gu, gc = Checkpointed(name, u0, T, C, slots=slots).backward(w, True)
    out.append((gu.clone(), gc))
for gu, gc in out[1:]:
    assert torch.equal(gu, out[0][0]), "grad_u0"
    assert torch.equal(gc, out[0][1]), (out[0][1], gc)
"""


@pytest.mark.parametrize("name", ["j2d5pt", "j2d9pt"])
@pytest.mark.parametrize("n", [1000, 2048])
@pytest.mark.parametrize("slots", ["1,8,1,8", "8,8,1"])
def test_bits_do_not_depend_on_earlier_launches(name, n, slots):
    env = dict(os.environ, PYTHONPATH=str(ROOT / "an5d-artifact_gb300"))
    r = subprocess.run([sys.executable, "-c", CHILD, name, str(n), slots], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
