"""Environment knobs that the integration notes list are read by the library; the
distances under the one of the narrow rows' rare counts."""
import os
import re
import subprocess
import sys

import pytest

from conftest import PKG_NAME, ROOT

PROG = """
import importlib, sys
sys.path[:0] = [%r, %r]
import numpy as np, torch
import oracle
pkg = importlib.import_module(%r)
A = np.random.default_rng(3).integers(0, 60, size=(900, 50)).astype(np.uint64)
want = np.triu(oracle.hamming(pkg.dense_ranks(A)[0]), 1)
with pkg.Solver.from_calls(A, tau=65536) as s:
    out = torch.zeros((900, 904), dtype=torch.int16, device="cuda")
    for rows in (899, 900):
        s.stripe(0, rows, out.data_ptr(), 904, torch.cuda.current_stream().cuda_stream)
        s.check()
        assert (np.triu(out[:rows, :900].cpu().numpy(), 1) == want[:rows]).all()
print("ok")
"""


def test_documented_knobs_are_read():
    with open(os.path.join(ROOT, "INTEGRATION.md")) as f:
        named = set(re.findall(r"TCH_[A-Z_]+", f.read()))
    with open(os.path.join(ROOT, "README.md")) as f:
        named |= set(re.findall(r"TCH_[A-Z_]+", f.read()))
    assert "TCH_RARE_SMALL_ROWS" in named
    read = set()
    for folder in ("csrc", "host", "."):
        d = os.path.join(ROOT, PKG_NAME, folder)
        for name in os.listdir(d):
            if name.endswith((".cu", ".cuh", ".cpp", ".h", ".py")):
                with open(os.path.join(d, name)) as f:
                    read |= set(re.findall(r"(?:getenv\(|environ[^\n]*)\"(TCH_[A-Z_]+)\"", f.read()))
    with open(os.path.join(ROOT, "include", "tch.h")) as f:
        header = set(re.findall(r"TCH_[A-Z_0-9]+", f.read()))
    missing = {k for k in named - header if k not in read} - {"TCH_LIB_DIR"}  # the Rust build script's own
    assert not missing, missing


@pytest.mark.gpu
@pytest.mark.parametrize("limit", ["0", "900"])
def test_distances_under_a_row_limit(limit):
    """No stripe, and only those of fewer than 900 rows, on the narrow rows' CTAs."""
    r = subprocess.run([sys.executable, "-c", PROG % (ROOT, os.path.join(ROOT, "oracle"), PKG_NAME)],
                       env={**os.environ, "TCH_RARE_SMALL_ROWS": limit}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-2000:]
