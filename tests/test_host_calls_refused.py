"""The library's host code over a stand-in for the CUDA runtime (tests/fake_cudart): what a call does when a launch or a copy
behind it is refused, and what its caller may do next."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from deepscalemd_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "deepscalemd_b200", "csrc")
CUDA_ERROR, CAPACITY, STATE = 2, 5, 6
i64, f64, ptr = ctypes.c_int64, ctypes.c_double, ctypes.c_void_p


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("fake_cudart")
    nvcc = build.nvcc_path()
    jobs = [subprocess.Popen([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-Xcicc", "-O0", "-std=c++17", "-ccbin", "/usr/bin/g++",
                              "-Xcompiler", "-fPIC", "-c", os.path.join(CSRC, f"{unit}.cu"), "-o", str(out / f"{unit}.o")])
            for unit in ("dsmd_core", "dsmd_edges")]
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-fPIC", "-c", "-x", "c++", "-I", include, "-I", CSRC, "-o", str(out / "fake.o"),
                    os.path.join(HERE, "fake_cudart", "fake_cudart.cpp")], check=True)
    assert all(job.wait() == 0 for job in jobs)
    subprocess.run(["/usr/bin/g++", "-shared", "-o", str(out / "libfake.so"), *(str(out / f"{n}.o") for n in ("dsmd_core", "dsmd_edges", "fake")),
                    "-Wl,-Bsymbolic", "-ldl"], check=True)
    lib = ctypes.CDLL(str(out / "libfake.so"))
    lib.fake_log.restype = ctypes.c_char_p
    return lib


@pytest.fixture(autouse=True)
def fresh(lib):
    lib.fake_reset()


def log(lib):
    return [lib.fake_log(k).decode() for k in range(lib.fake_log_size())]


# -- edge search: nothing may index with tables that a refused launch has not written ----------------------------------
@pytest.mark.parametrize("kernel,later", [("k_edge_keys", ("k_cell_starts", "k_edge_place", "k_edge_gather", "k_edge_search")),
                                          ("k_cell_sums", ("k_cell_starts", "k_edge_place", "k_edge_gather", "k_edge_search")),
                                          ("k_cell_starts", ("k_edge_place", "k_edge_gather", "k_edge_search")),
                                          ("k_edge_place", ("k_edge_gather", "k_edge_search")),
                                          ("k_edge_gather", ("k_edge_search",))])
@pytest.mark.parametrize("n,L", [(500, 100.0), (40000, 200.0)])   # tables that one launch scans, and two
def test_edge_search_ends_at_the_first_refused_launch(lib, kernel, later, n, L):
    if kernel == "k_cell_sums" and n < 40000:
        return   # one launch
    edges = ptr()
    assert lib.dsmd_edges_create(0, ctypes.byref(edges)) == 0
    x, box, n_edges = np.random.default_rng(1).uniform(0.0, L, (3, n)), np.full(3, L), i64()
    lib.fake_refuse(kernel.encode(), 0)
    rc = lib.dsmd_edges_build_periodic(edges, *(ptr(a.ctypes.data) for a in x), i64(n), ptr(box.ctypes.data), f64(5.0), ctypes.byref(n_edges), None)
    lines = log(lib)
    assert rc == CUDA_ERROR and any(line.startswith("refused") for line in lines)
    assert not [line for line in lines if any(k in line for k in later)]
    lib.fake_reset()   # the refusal is not reported a second time, and the next build starts with cleared counts
    lib.fake_refuse(b"k_edge_search", 0)
    lib.dsmd_edges_build_periodic(edges, *(ptr(a.ctypes.data) for a in x), i64(n), ptr(box.ctypes.data), f64(5.0), ctypes.byref(n_edges), None)
    assert any("k_edge_gather" in line for line in log(lib))
    lib.dsmd_edges_destroy(edges)
