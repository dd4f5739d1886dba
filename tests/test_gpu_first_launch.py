"""A process's first field step loads the device code it needs and no more."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes as C, sys, time
import torch
from oncolytica_b200 import _lib
olc, storage = _lib.load(), int(sys.argv[1])
kind = [torch.float32, torch.bfloat16, torch.float16, torch.bfloat16, torch.float16][storage]
ptr = lambda t: C.c_void_p(t.data_ptr())
def step(substeps):
    f = torch.full((64, 64, 64), 0.5, device="cuda", dtype=kind)
    tmp, comp = torch.zeros_like(f), torch.zeros(f.shape, device="cuda")
    spec = _lib.OlcDiffusion(diffusion=1.0, decay=0.05, boundary=0.7, substeps=substeps, storage=storage)
    dims = (C.c_int32 * 3)(64, 64, 64)
    torch.cuda.synchronize()
    t = time.perf_counter()
    if storage:
        rc = olc.olc_stage_diffuse16(ptr(f), ptr(tmp), None, ptr(comp), C.byref(dims), 1.0, 0.1 * substeps,
                                     C.byref(spec), 0, 0, None)
    else:
        rc = olc.olc_stage_diffuse(ptr(f), ptr(tmp), None, C.byref(dims), 1.0, 0.1 * substeps, C.byref(spec), None)
    torch.cuda.synchronize()
    assert rc == 0
    return time.perf_counter() - t
step(3)
print(step(20))
"""


@pytest.mark.parametrize("storage", [0, 4])
def test_first_resident_step_loads_little(cuda, storage):
    """64^3 after a field step by passes: 2 ms of it are the kernel's device code.  The
    limit is 10 ms, in the better of three processes."""
    took = []
    for _ in range(3):
        out = subprocess.run([sys.executable, "-c", SCRIPT, str(storage)], cwd=REPO, capture_output=True, text=True,
                             env=dict(os.environ, PYTHONPATH=REPO), timeout=300)
        assert out.returncode == 0, out.stderr
        took.append(float(out.stdout.split()[-1]))
    assert min(took) < 10e-3, took
