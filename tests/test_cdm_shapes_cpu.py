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


# (x, y, z): the grids of templates and subjects, long and flat volumes, rows of a few voxels
DIMS = [(91, 109, 91), (182, 218, 182), (128, 128, 128), (68, 66, 70), (4, 4, 20000), (8, 8, 5000), (16, 16, 1500),
        (24, 24, 800), (36, 32, 400), (1, 300, 300), (2, 300, 300), (3, 300, 300), (300, 300, 3), (300, 1, 1000),
        (200000, 1, 1), (1, 200000, 1), (2, 200000, 1), (1, 1, 200000), (1, 300, 1000)]


@pytest.mark.parametrize("dims", DIMS)
def test_poisson_threads_have_work(shapes, dims):
    """The sweeps' threads have places for at most twice the padded voxels (four a place), but for
    a block a component; and padded rows take at most 60 % more than their voxels (5 of 8)."""
    pitch, plane, _, pnb, pdz = shapes("dims", *dims)[:5]
    assert pnb * 256 * max(pdz, 1) <= 2 * 3 * (plane / 4) + 3 * 256 * max(pdz, 1)
    n = dims[0] * dims[1] * dims[2]
    assert plane <= 1.6 * n and pitch * dims[1] * dims[2] == plane


@pytest.mark.parametrize("dims", DIMS)
def test_tail_blocks_have_work(shapes, dims):
    """The tail launches have a block for each 512 places of a component."""
    plane, tnb = (shapes("dims", *dims)[k] for k in (1, 5))
    assert 512 * (tnb - 1) < plane <= 512 * tnb


@pytest.mark.parametrize("dims", DIMS)
def test_float_gradient_tiles_are_filled(shapes, dims):
    """The float gradient's tiles are kept where a quarter of their voxels, at least, are the
    volume's; ordinary grids keep them."""
    each = shapes("dims", *dims)[6]
    n = dims[0] * dims[1] * dims[2]
    depth = 2 if n < 200000 else 4
    tiles = -(-dims[0] // 32) * -(-dims[1] // 8) * -(-dims[2] // depth)
    assert each or 4 * n > tiles * 32 * 8 * depth
    assert not (each and min(dims) >= 36)


@pytest.mark.parametrize("dims", DIMS + [(300, 1, 300), (300, 2, 300), (23, 28, 23), (46, 55, 46)])
def test_uint8_gradient_tile_depth(shapes, dims):
    """The uint8 gradient's tiles are no deeper than the volume needs, and those of 2 planes are
    few enough for the blocks that share them."""
    nblk, shallow = (shapes("dims", *dims)[k] for k in (2, 7))
    tiles = -(-dims[0] // 32) * -(-dims[1] // 8) * -(-dims[2] // 2)
    assert shallow or dims[2] > 2
    assert not shallow or dims[2] <= 2 or tiles <= 3 * min(nblk, 444)
    assert shallow == 1 if dims in ((23, 28, 23), (46, 55, 46)) else True
