"""The library's host code over a stand-in for the CUDA runtime (tests/fake_cudart): what a call does when a launch or a copy
behind it is refused, and what its caller may do next; and which launches it makes."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from deepscalemd_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "deepscalemd_b200", "csrc")
CUDA_ERROR, OUT_OF_DOMAIN, CAPACITY, STATE = 2, 4, 5, 6
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


# -- list builds that fail ----------------------------------------------------------------------------------------------
class System:
    def __init__(self, lib, n=4000, L=16.8):
        self.lib, self.n, self.h = lib, n, ptr()
        assert lib.dsmd_create(0, i64(n), ctypes.byref(self.h)) == 0
        box, periodic, zero = np.full(3, L), (ctypes.c_int * 3)(1, 1, 1), np.zeros(3)
        assert lib.dsmd_set_box(self.h, *(ptr(a.ctypes.data) for a in (box,)), periodic, ptr(zero.ctypes.data), ptr(zero.ctypes.data), f64(0.0)) == 0
        one = np.ones(1)
        assert lib.dsmd_set_pair_params(self.h, ctypes.c_int(1), ptr(one.ctypes.data), ptr(one.ctypes.data), f64(2.5), f64(0.3), f64(-1.0)) == 0
        self.rows = np.random.default_rng(2).uniform(0.0, L, (n, 3))
        assert lib.dsmd_upload_rows(self.h, i64(n), i64(n), ptr(self.rows.ctypes.data), None, None, None, None, None, None) == 0

    def build(self):
        return self.lib.dsmd_build_neighbor_list(self.h, None)

    def forces(self):
        return self.lib.dsmd_compute_forces(self.h, ctypes.c_int(0), ctypes.c_int(0), None)

    def run(self, steps, every):
        return self.lib.dsmd_run_nve(self.h, i64(steps), f64(0.001), f64(1.0), f64(0.5), ctypes.c_int(every), ctypes.c_int(0), None, None, None)

    def displacement(self):
        return self.lib.dsmd_max_displacement_sq(self.h, ctypes.byref(f64()), None)


@pytest.fixture
def system(lib):
    s = System(lib)
    assert s.build() == 0 and s.forces() == 0
    yield s
    lib.dsmd_destroy(s.h)


def assert_no_list_until_rebuilt(s):
    assert s.forces() == STATE
    assert s.displacement() != CUDA_ERROR   # no wait for a check that a closed gate kept from reporting
    s.lib.fake_reset()
    assert s.build() == 0 and s.forces() == 0 and s.run(5, 2) == 0


@pytest.mark.parametrize("in_loop", [False, True])
@pytest.mark.parametrize("stride,outside,code", [(0xFFFFFFFF, 0, CAPACITY), (0, 1, OUT_OF_DOMAIN)])
def test_a_failed_build_leaves_no_list(lib, system, in_loop, stride, outside, code):
    """Rows that keep overflowing, an atom outside: the atoms have been sorted and the rows rewritten."""
    lib.fake_build_finds(ctypes.c_uint(stride), outside)
    assert (system.run(6, 2) if in_loop else system.build()) == code
    assert_no_list_until_rebuilt(system)


@pytest.mark.parametrize("kernel", ["k_cell_keys", "k_cell_starts", "k_place", "k_reorder", "k_build_rows", "k_build_done"])
def test_a_build_with_a_refused_launch_leaves_no_list(lib, system, kernel):
    lib.fake_refuse(kernel.encode(), 0)
    assert system.build() == CUDA_ERROR
    assert_no_list_until_rebuilt(system)


@pytest.mark.parametrize("kernel", ["k_step", "k_post_displacement"])
def test_a_step_refused_behind_a_build_leaves_no_list(lib, system, kernel):
    lib.fake_refuse(kernel.encode(), 1)   # the first one is in front of the build
    assert system.run(6, 2) == CUDA_ERROR
    lines = log(lib)
    assert "k_build_done" in "".join(lines[-3:]) and "refused" in lines[-1]
    assert_no_list_until_rebuilt(system)


def test_a_check_that_finds_an_atom_outside_can_be_asked_again(lib, system):
    lib.fake_check_finds(1)
    assert system.run(6, 0) == OUT_OF_DOMAIN
    assert system.displacement() != CUDA_ERROR


@pytest.mark.parametrize("positions_only", [False, True])
def test_a_sort_of_the_owned_atoms_does_not_count_for_atoms_uploaded_since(lib, system, positions_only):
    """A build behind dsmd_sort_owned sorts the ghosts alone: not if there are other atoms, or places, than were sorted."""
    assert lib.dsmd_sort_owned(system.h, None) == 0
    if positions_only:
        assert lib.dsmd_upload_positions(system.h, *(ptr(a.ctypes.data) for a in np.ascontiguousarray(system.rows.T)), None) == 0
    else:
        assert upload(system, system.rows) == 0
    lib.fake_reset()
    assert system.build() == 0
    assert any("k_cell_keys" in line for line in log(lib)) and any("k_reorder" in line for line in log(lib))


# -- uploads of rows ----------------------------------------------------------------------------------------------------
def upload(s, pos, vel=None):
    return s.lib.dsmd_upload_rows(s.h, i64(len(pos)), i64(len(pos)), ptr(pos.ctypes.data), ptr(vel.ctypes.data) if vel is not None else None, None,
                                  None, None, None, None)


@pytest.mark.parametrize("first,last", [(400, 600), (0, 1000), (0, 500), (500, 1000), (666, 667), (999, 1000)])   # registered: thousandths of the buffer
def test_rows_in_memory_registered_in_part(lib, first, last):
    """The runtime only queues a copy that starts in memory that it knows, and refuses it if the memory ends before; the call promises
    the rows back, of any memory."""
    n = 50000
    s = System(lib, n, 40.0)
    pos = np.random.default_rng(3).uniform(0.0, 40.0, (n, 3))
    lib.fake_reset()
    lib.fake_pin(ptr(pos.ctypes.data + pos.nbytes // 1000 * first), ctypes.c_size_t(pos.nbytes // 1000 * (last - first)))
    assert upload(s, pos) == 0
    lines = log(lib)
    queued = [k for k, line in enumerate(lines) if line == "queued copy"]
    assert not queued or "wait" in lines[queued[-1]:]
    lib.dsmd_destroy(s.h)


@pytest.mark.parametrize("fails", [1, 2, 4])
def test_rows_are_waited_for_when_a_later_copy_fails(lib, fails):
    s = System(lib, 50000, 40.0)
    pos = np.random.default_rng(4).uniform(0.0, 40.0, (50000, 3))
    lib.fake_reset()
    lib.fake_pin(ptr(pos.ctypes.data), ctypes.c_size_t(pos.nbytes))
    lib.fake_fail_copy(fails)
    assert upload(s, pos, pos) == CUDA_ERROR
    assert log(lib)[-1] == "wait"
    lib.dsmd_destroy(s.h)


# -- launches -----------------------------------------------------------------------------------------------------------
def test_no_report_of_a_check_whose_word_the_caller_has(lib):
    """Whoever has the displacement word's address reads it there (the loop over several GPUs): nothing is launched, or waited for
    within a kernel, for a report that nobody looks at; the loop of one GPU still reads its own."""
    s = System(lib, 30000, 33.0)
    assert s.build() == 0 and s.forces() == 0

    def launches_of_a_step():
        lib.fake_reset()
        assert lib.dsmd_integrate(s.h, ctypes.c_int(1), f64(0.001), f64(1.0), None) == 0
        return [line for line in log(lib) if line.startswith("launch")]

    assert [("k_pack" in line, "k_post_displacement" in line) for line in launches_of_a_step()] == [(True, False), (False, True)]
    word = ptr()
    assert lib.dsmd_displacement_word(s.h, ctypes.byref(word)) == 0
    for _ in range(2):
        lines = launches_of_a_step()
        assert len(lines) == 1 and "k_pack" in lines[0]
        assert s.displacement() == 0
        assert s.run(4, 2) == 0 and any("k_post_displacement" in line for line in log(lib))
    lib.dsmd_destroy(s.h)


@pytest.mark.parametrize("before", ["nothing", "no boundary pairs", "a refused launch", "another stream"])
def test_the_list_is_read_early_only_behind_a_force_launch(lib, before):
    """A force kernel reads the list before the launch before it has ended if a force launch of the same stream came between the list
    build and it: one that was made."""
    s = System(lib)
    assert s.build() == 0
    if before == "no boundary pairs":
        assert lib.dsmd_compute_forces(s.h, ctypes.c_int(2), ctypes.c_int(0), None) == 0   # nothing to launch
    if before == "a refused launch":
        lib.fake_refuse(b"k_pair", 0)
        assert s.forces() == CUDA_ERROR
    if before == "another stream":
        assert lib.dsmd_compute_forces(s.h, ctypes.c_int(0), ctypes.c_int(0), ptr(64)) == 0
    lib.fake_reset()
    assert s.forces() == 0 and s.forces() == 0
    assert [line for line in log(lib) if "k_pair" in line] == ["launch k_pair", "launch k_pair early"]
    lib.dsmd_destroy(s.h)
