"""Functors derived from the bundled ones (tests/dropin/override_functors.cu):
which extensions a derived functor keeps is checked when it compiles, and the
GPU test runs a BFS whose overridden combine offers two levels per hop, by the
hybrid policy and by pull rounds alone, against twice the oracle's levels."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle
import sepgraph as sg

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sep-graph_b200")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    sg.load()  # the library must be built
    out = str(tmp_path_factory.mktemp("overrides") / "override_functors")
    cmd = [NVCC, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
           "-Xcudafe", "--diag_suppress=esa_on_defaulted_function_ignored", "-Xptxas", "-dlcm=cg",
           "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "dropin", "override_functors.cu"), "-o", out,
           "-L", PKG, "-lsepgraph_b200", "-Xlinker", "-rpath", "-Xlinker", PKG]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return out


def test_overrides_select_extensions(exe):
    assert os.path.exists(exe)


@pytest.mark.gpu
def test_overridden_combine_runs_in_pull_rounds(exe, tmp_path):
    h = sg.HostGraph.rmat(13, 16, symmetric=True, seed=1)
    root = int(h.max_degree_vertex()[0])
    prefix = str(tmp_path / "out")
    r = subprocess.run([exe, "13", str(root), prefix], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    levels = oracle.bfs(h.offsets, h.indices, root)
    want = np.where(levels == 0xFFFFFFFF, levels, 2 * levels)
    for name in ("hybrid", "pull"):
        assert np.array_equal(np.fromfile(f"{prefix}_{name}.u32", dtype=np.uint32), want), name
