"""The batched schedules' time blocks (csrc/batch_blocks.h, compiled and run
here): every split of T = 1..200 steps for every pair of a layered and a
persistent degree sums to T, has T's parity of blocks and no empty block,
stays within the layered degree, and ends an odd T with the persistent
schedule's last block."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "an5d-artifact_gb300" / "csrc"

MAIN = r"""
#include "batch_blocks.h"
#include <cstdio>
static void show(const std::vector<int> &v) {
  for (size_t i = 0; i < v.size(); ++i) std::printf("%s%d", i ? "," : "", v[i]);
}
int main() {
  for (int p = 1; p <= 6; ++p)
    for (int b = p; b <= 6; ++b)
      for (int T = 0; T <= 200; ++T) {
        std::printf("%d %d %d ", p, b, T);
        show(gbs::batch_blocks(T, p));
        std::printf(";");
        show(gbs::layered_blocks(T, b, p));
        std::printf("\n");
      }
}
"""


@pytest.fixture(scope="module")
def splits(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("blocks")
    (d / "main.cc").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(CSRC), str(d / "main.cc"), "-o", str(d / "main")], check=True)
    out = subprocess.run([str(d / "main")], capture_output=True, text=True, check=True).stdout
    parse = lambda s: [int(x) for x in s.split(",")] if s else []
    rows = []
    for line in out.splitlines():
        head, layered = line.split(";")
        p, b, T, *rest = head.split(" ")
        rows.append((int(p), int(b), int(T), parse(rest[0]), parse(layered)))
    return rows


def test_blocks_of_every_length_and_degree(splits):
    assert len(splits) == 21 * 201
    for p, b, T, persistent, layered in splits:
        for blocks, top in ((persistent, p), (layered, b)):
            assert sum(blocks) == T and len(blocks) % 2 == T % 2, (p, b, T, blocks)
            assert all(1 <= x <= top for x in blocks), (p, b, T, blocks)
        assert set(persistent) <= {p, 1}
        if T % 2:
            assert layered[-1] == persistent[-1], (p, b, T)
