"""Launch decisions of the CDM passes that need no device: the compiled passes linked with a
stand-in for the CUDA runtime (tests/cpp/cdm_shapes.cpp)."""
import os
import subprocess

import pytest

from tipl_b200 import build as b

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    b.build()
    obj = os.path.join(b.BUILD, "cdm_kernels.cu.o")
    if not os.path.exists(obj):
        b.build(force=True)
    exe = str(tmp_path_factory.mktemp("cdm_shapes") / "cdm_shapes")
    subprocess.check_call(["g++", "-std=c++17", "-I", b.CSRC, "-I", b.INCLUDE, "-I", f"{b.CUDA_HOME}/include",
                           os.path.join(ROOT, "tests", "cpp", "cdm_shapes.cpp"), obj, "-o", exe])
    return lambda *a: [int(v) for v in subprocess.check_output([exe, *map(str, a)], text=True).split()]


def test_failed_cluster_check_leaves_no_error(shapes):
    """Where a call of the cluster check fails, the sweeps run without clusters, and no error
    stays behind for the next launch to report."""
    used, error, calls = shapes("probe", 0)
    assert (used, error) == (1, 0) and calls > 1
    for k in range(1, calls + 1):
        assert shapes("probe", k)[:2] == [0, 0]
