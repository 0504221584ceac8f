"""Persistent solves on both sides of the rules that choose their thread-block clusters: one
cluster of 8, one of 16 (from 9 blocks' worth of nodes to 31), several clusters of which the first
runs the coarse levels (up to three FP64 or four FP32 level-1 nodes a thread of it), and grids
without clusters, with odd row lengths.  The checks are those of the layout's shapes: the
reference's stop rules, recomputed in numpy."""
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

import semiconductor_devices_simulator_b200 as S  # noqa: E402
import test_gpu_persist_shapes as P  # noqa: E402

pytestmark = pytest.mark.gpu
# blocks' worth (1024 nodes each): 8, 9, 16, 31, 32; level-1 nodes 24,192 and 25,056 (the FP64
# limit is 24,576), 32,736 and 33,792 (the FP32 limit is 32,768)
SHAPES = [(64, 16, 8), (33, 19, 14), (31, 27, 19), (37, 31, 27), (33, 32, 31), (63, 55, 54), (71, 57, 48), (61, 66, 64),
          (63, 64, 65)]


@pytest.fixture(scope="module")
def lib():
    return S.load()


@pytest.fixture(params=[0, 1], ids=["fp64", "refined"])
def precision(lib, request):
    old = lib.api3b_set_precision(request.param)
    yield request.param
    lib.api3b_set_precision(old)


@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
def test_persistent_clusters(lib, precision, n):
    P.test_persistent_bicgstab_shapes(lib, precision, n)
    P.test_persistent_pcg_shapes(lib, precision, n)
