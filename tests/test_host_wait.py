"""The host's wait for a product's state (gpuspgemm_b200/csrc/host_wait.hpp).

CPU: the wait itself, with a thread in the device's place: how it waits follows
the process's schedule, the stream is asked at most once per interval, and a
stream that failed or ended without the flag ends the wait.  GPU: a process that
asked for blocking waits sleeps in them."""
import json
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def wait_bin(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = tmp_path_factory.mktemp("wait") / "host_wait_host"
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", str(HERE / "host_wait_host.cpp"),
                    "-o", str(out)], check=True, timeout=120)
    return out


def run(wait_bin, schedule, ms, end, raised):
    res = subprocess.run([str(wait_bin), schedule, str(ms), str(end), str(raised)],
                         capture_output=True, text=True, check=True, timeout=60)
    return json.loads(res.stdout)


@pytest.mark.parametrize("schedule", ["spin", "yield", "block"])
@pytest.mark.parametrize("ms", [0, 1, 20])
def test_raised(wait_bin, schedule, ms):
    r = run(wait_bin, schedule, ms, 1, 1)
    assert r["end"] == "raised"
    assert r["queries"] <= r["us"] / r["query_us"], r
    assert r["blocks"] == (schedule == "block"), r
    assert (r["yields"] > 0) <= (schedule == "yield"), r
    if ms == 20:
        assert (r["yields"] > 0) == (schedule == "yield"), r


@pytest.mark.parametrize("schedule", ["spin", "yield", "block"])
@pytest.mark.parametrize("end,raised,want", [(-1, 0, "failed"), (-1, 1, None), (1, 0, "not raised")])
def test_stream_ends(wait_bin, schedule, end, raised, want):
    r = run(wait_bin, schedule, 2, end, raised)
    # (a flag that is up tells that the stream's earlier work is done)
    assert r["end"] == want if want else r["end"] in ("raised", "failed"), r


CHILD = """
import ctypes, sys, time
sys.path.insert(0, sys.argv[1])
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
flags = {"spin": 1, "yield": 2, "block": 4}[sys.argv[2]]
assert cu.cuDevicePrimaryCtxSetFlags_v2(0, flags) == 0
import torch
from gpuspgemm_b200 import generators as G
from gpuspgemm_b200.api import DeviceCSR, Handle, proposal
torch.cuda.set_device(0)
A = DeviceCSR.from_host(G.uniform_rows(200_000, 16, seed=3))
h = Handle(0)
ref = proposal(A, A, h)
for _ in range(5):
    proposal(A, A, h)
torch.cuda.synchronize()
t, c = time.perf_counter(), time.thread_time()
for _ in range(50):
    C = proposal(A, A, h)
wall, cpu = time.perf_counter() - t, time.thread_time() - c
assert torch.equal(C.rpt, ref.rpt) and torch.equal(C.col, ref.col)
print("SHARE", cpu / wall)
"""


@pytest.mark.gpu
@pytest.mark.parametrize("schedule", ["spin", "yield", "block"])
def test_process_schedule(native_lib, schedule):
    res = subprocess.run([sys.executable, "-c", CHILD, str(HERE.parent), schedule],
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    share = float(res.stdout.split("SHARE")[1])
    # this product computes for over a millisecond and its host work is ~0.3 ms
    if schedule == "block":
        assert share < 0.75, share
