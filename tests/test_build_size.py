"""The build's objects and library stay small enough to move with the tree
(line tables alone once made them 290 MB each)."""
import pytest

from gbstencil import build


def test_build_outputs_stay_small():
    if not build.LIB.exists():
        pytest.skip("not built")
    objects = [build.BUILD / f"{u[0]}.o" for u in build.units()]
    total = build.LIB.stat().st_size + sum(o.stat().st_size for o in objects if o.exists())
    assert total < 256 << 20, f"{total >> 20} MiB of build outputs"
