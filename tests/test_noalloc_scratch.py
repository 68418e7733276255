"""The allocation-free transform's device array: the library holds the 64 MiB it states
and no more (as ptxas reports the global memory of its translation unit; the FFT's
constant tables may add a few KiB), and the twiddle tables inside it serve every
kind of length: compiled plans of both variants and run-time plans, on each axis."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from tests.problems import ROOT


def test_scratch_is_the_stated_size(tmp_path):
    from coral_b200 import build
    src = os.path.join(ROOT, "coral_b200", "csrc", "noalloc.cu")
    r = subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-Xptxas", "-v", "-cubin", "-o", str(tmp_path / "n.cubin"),
                        src], capture_output=True, text=True, check=True)
    gmem = int(re.search(r"(\d+) bytes gmem", r.stderr + r.stdout).group(1))
    assert 64 << 20 <= gmem <= (64 << 20) + 4096


# 576 points along x, y, z; merged plans (486, 108, 162, 324, 432); run-time lengths 6, 12, 18
@pytest.mark.gpu
@pytest.mark.parametrize("N", [(384, 4, 8), (4, 384, 4), (8, 4, 384), (324, 12, 16), (72, 108, 216), (16, 288, 72),
                               (128, 128, 96)])
def test_every_kind_of_length(N):
    import torch
    from coral_b200 import _lib
    from oracle import coral_oracle as co
    lib = _lib.load()
    torch.cuda.set_device(0)
    g = co.Geometry(*N, 2.0, 3.0, 1.0, 0.5)
    rng = np.random.default_rng(5)
    spec = rng.standard_normal((g.NXH, g.NYAA, g.NZ)) + 1j * rng.standard_normal((g.NXH, g.NYAA, g.NZ))
    ref = co.spec_to_phys(spec, g)
    d_spec = torch.from_numpy(spec.view(np.float64).ravel()).cuda()
    d_phys = torch.full(ref.shape, float("nan"), dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))
    assert lib.coral_spec_to_phys_noalloc(*N, p(d_spec), p(d_phys), None) == 0, lib.coral_last_error(None).decode()
    torch.cuda.synchronize()
    # same tolerance as the transform parity tests
    assert np.abs(d_phys.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
