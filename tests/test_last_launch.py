"""Loops of odd T: plane T%2 holds u_T, and the other plane the state before
the last launch, whose steps the table's "last" degree fixes whatever degree
the loop runs at (a program that runs such a loop again starts from it)."""
import numpy as np
import pytest

import pyoracle as po
from gbstencil import capi, tune


@pytest.fixture
def table(tmp_path):
    capi.lib()
    saved = tmp_path / "saved.txt"
    tune.save(saved)
    tune.clear()
    yield tmp_path / "t.txt"
    tune.clear()
    tune.load(saved)


def launches(T, bt):
    d, _ = capi.make_desc("star2d1r", np.float32, 100, T, "exact")
    p = capi.plan(d)
    assert p.bt == bt
    return p.launches


def test_plan_counts_the_last_launch(table):
    table.write_text("star2d1r f32 exact 13 3 0 1.0\nstar2d1r f32 exact_last 13 2 0 0\n")
    tune.load(table)
    assert launches(12, 3) == 4
    assert launches(9, 3) == 5   # 8 steps in an even number of launches of at most 3, then 1
    tune.record("star2d1r", np.float32, 100, bt=3, fp_mode="exact")  # an entry recorded counts for both
    assert launches(9, 3) == 3
    again = table.with_suffix(".2")
    table.write_text("star2d1r f32 exact 13 3 0 1.0\nstar2d1r f32 exact_last 13 0 0 0\n")
    tune.load(table)
    tune.save(again)
    assert "star2d1r f32 exact_last 13 0 0 0" in again.read_text()


@pytest.mark.gpu
@pytest.mark.parametrize("T", [1, 3, 5, 9, 16, 31])
def test_plane_without_the_result(table, T):
    table.write_text("star2d1r f32 exact 13 4 0 1.0\nstar2d1r f32 exact_last 13 2 0 0\n")
    tune.load(table)
    A = po.init_grid("star2d1r", 100, np.float32)
    n = -(-T // 2)
    n += (n - T) % 2
    before = A.copy()
    po.run("star2d1r", before, 100, T - T // n if T % 2 else T)
    after = A.copy()
    po.run("star2d1r", after, 100, T)
    d, _ = capi.make_desc("star2d1r", np.float32, 100, T, "exact")
    capi.run_host(d, A)
    assert np.array_equal(A[T % 2], after[T % 2])
    if T % 2:
        assert np.array_equal(A[0], before[(T - T // n) % 2])


@pytest.mark.parametrize("bt,last", [(1, 2), (1, 4), (4, 1), (3, 2), (2, 4)])
def test_every_launch_takes_steps(table, bt, last):
    """The plan's launches keep T's parity and none is empty."""
    table.write_text(f"star2d1r f32 exact 13 {bt} 0 1.0\nstar2d1r f32 exact_last 13 {last} 0 0\n")
    tune.load(table)
    for T in range(1, 40):
        n = launches(T, bt)
        assert n % 2 == T % 2 and n <= T
