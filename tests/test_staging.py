"""Copies through the pinned staging: piece borders in both directions against a runtime of the test's own
(CPU; allocations, copies and threads that fail among them), and the same borders through the library."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pieces_and_failures_against_a_fake_runtime(tmp_path):
    exe = str(tmp_path / "staging")
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", os.path.join(ROOT, "tests", "staging_harness.cpp"), "-o", exe,
                    "-I/usr/local/cuda/include", "-I" + os.path.join(ROOT, "marvel_b200", "csrc"), "-pthread", "-ldl"],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n", [87381, 87382, 1048575, 1048576, 1048577, 1572864, 1572865, 1835009])
def test_piece_borders_through_mlp_forward(n):
    """48 n bytes up, 4 n bytes down (4 MB at 1,048,576): the same values as in calls too small to be staged."""
    import marvel_b200 as mb
    rng = np.random.default_rng(n)
    feat = rng.standard_normal((n, mb.TRI_NF), dtype=np.float32)
    params = rng.standard_normal(mb.TRI_NPARAM, dtype=np.float32) * np.float32(0.1)
    ctx = mb.Context()
    got = ctx.mlp_forward(params, feat)
    step = 32768
    want = np.concatenate([ctx.mlp_forward(params, feat[i:i + step]) for i in range(0, n, step)])
    ctx.close()
    assert np.array_equal(got, want)
