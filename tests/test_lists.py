"""CPU: the row lists' limits (gpuspgemm_b200/csrc/lists.hpp) and their bound: a
ladder with more limits than the scratch has lists is refused, not binned past
the end of the lists."""
import json
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent


@pytest.fixture(scope="module")
def lists_bin(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = tmp_path_factory.mktemp("lists") / "lists_host"
    subprocess.run([cxx, "-O1", "-std=c++17", f"-I{HERE / 'simt_host' / 'fake'}",
                    f"-I{ROOT / 'gpuspgemm_b200' / 'csrc'}", str(HERE / "lists_host.cpp"),
                    "-o", str(out)], check=True, timeout=120)
    return out


def run(lists_bin, nb, esc, min_bin=0):
    res = subprocess.run([str(lists_bin), str(nb), str(esc), str(min_bin)], capture_output=True,
                         text=True, check=True, timeout=60)
    return json.loads(res.stdout)


@pytest.mark.parametrize("nb,esc", [(8, 1), (9, 1), (10, 1), (13, 1), (9, 0), (12, 0), (13, 0), (16, 0)])
def test_bound(lists_bin, nb, esc):
    r = run(lists_bin, nb, esc)
    need = nb + (3 if esc else 0)
    assert r["ok"] == (need <= r["lists"]), r
    assert r["nb"] == (need if r["ok"] else -1), r


def test_limits_and_bins(lists_bin):
    r = run(lists_bin, 9, 1)
    assert r["limits"][:8] == [12, 48, 192, 512, 768, 1024, 2048, 3072]
    assert r["limits"] == sorted(r["limits"])
    assert r["hash_bin"] == [0, 1, 2, 3, 3, 4, 4, 4, 5, 6, 7, 8]
    assert r["sort_bin"] == [0, 1, 2, 3, 4, 4, 4, 4, 5, 6, 7, 8]


@pytest.mark.parametrize("min_bin,first", [(1, 1), (3, 3), (4, 5), (5, 8)])
def test_forced_bins(lists_bin, min_bin, first):
    r = run(lists_bin, 9, 1, min_bin)
    assert r["min"] == first and r["hash_bin"][first] == min_bin
