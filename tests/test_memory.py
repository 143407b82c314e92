"""Device memory that the library keeps between calls (the working pool, at most
512 MB) is given back before any of its allocations fails and is counted as free
where a decision hangs on free memory; the rest goes back when a call ends."""
import glob
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import PKG_NAME, ROOT

CSRC = os.path.join(ROOT, PKG_NAME, "csrc")


def test_every_device_allocation_takes_the_kept_memory_back():
    """The runtime's allocation calls and its free-memory query are made in one
    file, which retries; a page-locked host allocation is another matter."""
    calls = re.compile(r"\b(cudaMalloc|cudaMallocAsync|cudaMallocFromPoolAsync|cudaMemGetInfo)\(")
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.cpp"))):
        if os.path.basename(path) in ("memory.cpp", "peak.cu"):  # peak.cu: a program of its own
            continue
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        assert not calls.findall(text), os.path.basename(path)


def test_allocations_against_a_fake_runtime(tmp_path):
    include = next((d for d in ("/usr/local/cuda/include",) if os.path.exists(os.path.join(d, "cuda_runtime.h"))), None)
    if include is None:
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / "memory_check")
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-isystem", include, os.path.join(ROOT, "tests", "sanitize", "memory_check.cpp"),
                    os.path.join(CSRC, "memory.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "memory ok" in r.stdout, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["calls", "ranks", "database"])
def test_inputs_are_given_back_when_the_call_ends(pkg, how):
    """1.2 GB of calls: afterwards the device lacks what the object holds, and at
    most the kept 512 MB (and 128 MB for what else the runtime takes)."""
    torch = pytest.importorskip("torch")
    n, L = 100000, 1500
    A = np.zeros((n, L), np.uint16 if how == "ranks" else np.uint64)
    A[:, :4] = np.random.default_rng(1).integers(1, 9, size=(n, 4))
    make = {"calls": pkg.Solver.from_calls, "ranks": pkg.Solver.from_ranks, "database": pkg.Database}[how]
    make(A[:100], tau=4).close()  # the context and the kernels' modules
    free0 = torch.cuda.mem_get_info()[0]
    obj = make(A, tau=4)
    held = obj.info()["device_bytes"]
    lacks = free0 - torch.cuda.mem_get_info()[0] - held
    assert lacks < (512 + 128) << 20, (lacks, held)
    assert pkg.free_vram() >= torch.cuda.mem_get_info()[0]
    obj.close()
