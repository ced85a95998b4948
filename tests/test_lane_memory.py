"""A batch lane where device or page-locked memory runs out, on a device that is
not there (tests/host_cuda)."""
import os
import re
import shutil
import subprocess

import pytest

import qmetal_gb300 as qm

HERE = os.path.dirname(os.path.abspath(__file__))
OBJ = os.path.join(os.path.dirname(qm.library_path()), "_build")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def build_client(name, where):
    """tests/host_cuda/<name>.cpp with the host's objects and the device that is not there."""
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = str(where / name)
    r = subprocess.run(["gcc", "-w", "-c", os.path.join(HERE, "host_cuda", "fake_kernels.c"), "-o",
                        exe + ".kernels.o"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    cmd = ["g++", "-std=c++17", "-O1", "-w", "-pthread", "-I" + os.path.join(CUDA, "include")]
    cmd += [os.path.join(HERE, "host_cuda", f) for f in (name + ".cpp", "fake_device.cpp")]
    cmd += [os.path.join(OBJ, f + ".cpp.o") for f in ("simulator", "batch", "schedule", "plan", "circuit")]
    cmd.append(exe + ".kernels.o")
    r = subprocess.run(cmd + ["-o", exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]

    def run(what):
        out = subprocess.run([exe, what], capture_output=True, text=True, timeout=120)
        assert out.returncode == 0, out.stderr
        return {k: int(v) for k, v in re.findall(r"(\w+) (\d+)", out.stdout)}

    return run


@pytest.fixture(scope="module")
def client(tmp_path_factory):
    return build_client("lanes", tmp_path_factory.mktemp("lanes"))


def test_pinned_memory_fails(client):
    """The lanes then allocate for themselves, without the shared block beside them."""
    got = client("pinned")
    assert got["held"] == 0
    assert got["wide"] > 0 and got["narrow"] > 0
    assert got["left"] == 0


def test_no_second_buffer_for_the_widest(client):
    """Narrower requests that have room for theirs use the gather passes."""
    got = client("scratch")
    assert got["wide"] == 0
    assert got["narrow"] > 0
    assert got["left"] == 0


def test_memory_of_a_narrow_request(client):
    """A lane's phase tables and kept states lie beside the rest of its memory at each width."""
    got = client("narrow")
    assert got["small"] > 4 and got["overlaps"] == 0
    assert got["left"] == 0


def test_memory_of_a_simulator(client):
    """A narrow simulator holds its state, workspace and results, and what a gradient
    keeps from the first one on."""
    got = client("create")
    fixed = (8 << 12) + (1 << 20) + 8 * 4096
    assert got["made"] <= fixed and got["ran"] == got["made"]
    # the co-state, sixteen kept states and the gradient of 69 gates
    assert got["gradient"] <= fixed + 17 * (8 << 12) + 8 * 69
    assert got["small"] >= 2 and got["overlaps"] == 0
