"""Host-side logic that needs no GPU, compiled and run on the CPU: the sizes of the grid
reductions (hila_b200/csrc/hop_shapes.h) by tests/cpp/test_reductions.cpp, the division of the
engine's tiles (engine_parts.h) by test_parts.cpp, graph construction (graph_build.h) over a
fake CUDA runtime by test_graph_build.cpp, the cache of graphs (graph_cache.h) by
test_graph_cache.cpp, copies into pageable memory over a fake runtime by test_host_copy.cpp."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hila_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def compile_and_run(tmp_path, name, *flags):
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    exe = str(tmp_path / name)
    cc = subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC,
                         os.path.join(ROOT, "tests", "cpp", name + ".cpp"), *flags, "-o", exe],
                        capture_output=True, text=True)
    assert cc.returncode == 0, cc.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


def test_reduction_sizes(tmp_path):
    assert "reduction sizes passed" in compile_and_run(tmp_path, "test_reductions")


def test_parts(tmp_path):
    assert "parts passed" in compile_and_run(tmp_path, "test_parts")


def test_graph_build(tmp_path):
    assert "graph construction passed" in compile_and_run(tmp_path, "test_graph_build", "-I", CUDA_INCLUDE)


def test_graph_cache(tmp_path):
    assert "graph cache passed" in compile_and_run(tmp_path, "test_graph_cache")


def test_host_copy(tmp_path):
    assert "host copies passed" in compile_and_run(tmp_path, "test_host_copy", os.path.join(CSRC, "host_copy.cpp"),
                                                   "-I", CUDA_INCLUDE, "-pthread")
