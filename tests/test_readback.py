"""Results brought to pageable memory through the pinned ring equal those copied to pinned memory, around the ring's thresholds
(1, 16 and 32 MiB), its chunks (512 KiB) and more chunks than its slots (GPU); the ring over a stand-in for the CUDA runtime (CPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, grid

CUDA_INCLUDE = os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))), "include")


@pytest.fixture(scope="module")
def host_program(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime_api.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path_factory.mktemp("readback") / "readback_host")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-I", CUDA_INCLUDE,
                           os.path.join(ROOT, "tests", "c", "readback_host.cpp"),
                           os.path.join(ROOT, "olf-gpu_b200", "csrc", "readback.cpp"), "-pthread", "-ldl", "-o", exe])
    return exe


@pytest.mark.parametrize("case", ["pending", "own", "sizes", "pin", "event", "threads", "memory", "ways"])
def test_ring_over_a_stand_in_runtime(host_program, case):
    """A launch error from before the copy is still there after it, the copy's own failed calls leave none, and the bytes are
    the source's.  A ring, an event, a thread or memory that cannot be had: nothing is lost, and the copy is made all the
    same.  Arrays in memory are copied directly up to 32 MiB, and the ring is not pinned before the copies it is for add up to
    16 MiB."""
    out = subprocess.run([host_program, case], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 32, 33, 49, 131, 132, 1049])
def test_pageable_results_equal_pinned_ones(engine_lib, count):
    import torch
    from olfgpu import native, synthetic
    g, p = grid("grid2000")
    s = native.Structure(p, native.PLAN_DEFAULT)
    ctx = native.BatchContext(s, count)
    ctx.set_schedule(native.LEVELS_SHARED_ALL, 0, 256)
    dis = p.outage_masks(synthetic.draw_outages(g, count, seed=3))
    pinned = torch.empty((count, p.n + 3), dtype=torch.float64).pin_memory().numpy()
    ctx.solve(p.x_base, p.target, p.base_row_mode, dis, out=pinned)
    for _ in range(2):          # a small result's first copy is direct
        fresh = ctx.solve(p.x_base, p.target, p.base_row_mode, dis)
        assert np.array_equal(fresh, pinned, equal_nan=True)
    kept = []                   # fresh arrays, through the ring once they add up to 16 MiB
    for _ in range(0 if count > 500 else 18):
        kept.append(ctx.solve(p.x_base, p.target, p.base_row_mode, dis))
        assert np.array_equal(kept[-1], pinned, equal_nan=True)


@pytest.mark.gpu
def test_security_analysis_writes_chunks_in_place(engine_lib):
    """A last chunk shorter than the others is padded and copied; every row equals the single batch's."""
    from olfgpu import synthetic
    from olfgpu.security_analysis import SecurityAnalysis
    g, p = grid("grid118")
    outs = synthetic.draw_outages(g, 50, seed=4)
    sa = SecurityAnalysis(p)
    whole, parts = sa.solve_n1(outs), sa.solve_n1(outs, chunk=16)
    assert np.array_equal(whole.x, parts.x) and np.array_equal(whole.status, parts.status)
