"""Pages that a thread makes ahead of a copy to the host (csrc/pages.h).  The thread has no device of its own, so its code makes
no CUDA call: it is built and linked here without CUDA's headers and runtime."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_pages_are_made_without_cuda(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no C++ compiler"
    exe = str(tmp_path / "pages")
    subprocess.check_call([cxx, "-std=c++17", "-O1", "-pthread", os.path.join(ROOT, "tests", "cpp", "pages.cpp"),
                           "-I", os.path.join(ROOT, "tsne_cuda_b200", "csrc"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["fresh", "off by four bytes", "pinned", "device", "one of each"])
def test_lists_in_any_memory(engine, where):
    """Lists of 2.4 MB, whose pages a thread makes while the search runs, where it may."""
    import ctypes as C

    import torch
    n, d, k = 20000, 8, 30
    X = np.random.default_rng(5).normal(0, 1, (n, d)).astype(np.float32)
    want_i, want_d = engine.knn(X, k)

    def array(kind, dtype):
        if kind == "pinned":
            return torch.empty(n * k, dtype=getattr(torch, dtype)).pin_memory()
        if kind == "device":
            return torch.empty(n * k, dtype=getattr(torch, dtype), device="cuda")
        if kind == "off by four bytes":
            return np.empty(n * k + 1, dtype)[1:]
        return np.empty(n * k, dtype)

    ids = array("device" if where == "one of each" else where, "int32")
    d2 = array("fresh" if where == "one of each" else where, "float32")
    torch.cuda.synchronize()
    at = [a.data_ptr() if torch.is_tensor(a) else a.ctypes.data for a in (ids, d2)]
    engine.check(engine.lib.b200tsne_knn(engine._f(X), n, d, k, 0, n, 0, n, C.cast(at[0], C.POINTER(C.c_int32)),
                                         C.cast(at[1], C.POINTER(C.c_float)), 0))
    torch.cuda.synchronize()
    assert np.array_equal(torch.as_tensor(ids).cpu().numpy().reshape(n, k), want_i)
    assert np.array_equal(torch.as_tensor(d2).cpu().numpy().reshape(n, k), want_d)
