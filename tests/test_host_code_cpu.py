"""Host code of the library on a stand-in CUDA runtime (tests/native/fake_cuda.h), whose calls can be
told to fail: no device is needed, and none is asked to fail."""
import os
import subprocess

import pytest

from solidfem_b200 import build as b

NATIVE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native")


def program(folder, name):
    """tests/native/<name>.cpp, with the library's <name>.cpp where there is one."""
    out = str(folder / name)
    library = os.path.join(b.CSRC, name + ".cpp")
    subprocess.run([b.CXX, "-std=c++17", "-O1", "-fopenmp", "-Wno-unused-function", "-I" + NATIVE, "-I" + b.CSRC,
                    "-I" + os.path.join(b.CUDA, "include"), os.path.join(NATIVE, name + ".cpp"),
                    *([library] if os.path.exists(library) else []), "-o", out],
                   check=True, capture_output=True, text=True)
    return out


def run(*command):
    r = subprocess.run([str(c) for c in command], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.fixture(scope="module")
def host_link(tmp_path_factory):
    return program(tmp_path_factory.mktemp("host_link"), "host_link")


@pytest.mark.parametrize("pinned", ["pinned", "no-pinned", "one-pinned"])
@pytest.mark.parametrize("size", [0, 8, (64 << 10) - 8, 64 << 10, (4 << 20) + 8, 9 << 20])
def test_arrays_cross_whether_or_not_page_locked_memory_is_to_be_had(host_link, pinned, size):
    run(host_link, pinned, size)


@pytest.mark.parametrize("size", [8, (64 << 10) - 8, 64 << 10, 9 << 20])
def test_a_load_vector_may_be_reused_once_it_was_taken(host_link, size):
    run(host_link, "reuse", size)


@pytest.mark.parametrize("size", [88, 176, 264, 2112])
def test_a_small_array_may_cross_in_smaller_chunks(host_link, size):
    run(host_link, "small-chunks", size)


@pytest.fixture(scope="module")
def iterations(tmp_path_factory):
    return program(tmp_path_factory.mktemp("iterations"), "iterations")


@pytest.mark.parametrize("case", ["whole", "no-instantiation", "no-capture", "no-launch"])
def test_a_solve_does_not_need_its_longer_graph(iterations, case):
    run(iterations, case)


@pytest.mark.parametrize("case", ["soon-over", "long-enough", "long", "short-solves"])
def test_the_longer_graph_is_made_where_it_pays(iterations, case):
    """5 kernels an iteration: worth 80 iterations. Looked at from iteration 12 on, a solve of 90 has 78
    to go and does not make it, solves of 100 and 211 do. 14 kernels: worth 224, the sixth solve of 39
    has seen 195, the seventh more."""
    run(iterations, case)


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    return program(tmp_path_factory.mktemp("rules"), "rules")


@pytest.mark.parametrize("lanes,rows,longest,expected", [
    (4, 30375, 7, 8), (4, 1000, 256, 8), (4, 1000, 257, 32), (4, 8192, 1000, 32), (4, 8193, 1000, 8),
    (8, 1000, 1000, 8), (16, 1000, 7, 16), (32, 30375, 7, 32)])
def test_lanes_of_short_rows_and_of_a_few_long_ones(rules, lanes, rows, longest, expected):
    assert int(run(rules, "product_lanes", lanes, rows, longest)) == expected
