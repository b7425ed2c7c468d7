"""The autotuner changes only what the batch at hand reads, and sort_min is
taken as it is set."""
import ctypes

import numpy as np
import pytest
import torch

from distance3d_gb300 import _lib, workloads
from distance3d_gb300.serve import CollisionBatch
from distance3d_gb300.store import ColliderStore
from distance3d_gb300.tune import autotune, get_tuning, set_tuning

pytestmark = pytest.mark.gpu


@pytest.fixture
def scene():
    before = get_tuning()
    cs, i1, i2 = workloads.pairs_mixed_six(9000, seed=51, center_half_width=workloads.INTERSECT30_HALF_WIDTH)
    yield ColliderStore(cs), np.asarray(i1, np.int32), np.asarray(i2, np.int32)
    set_tuning(**before)


def sort_kernels(st, n):
    """The toolkit's (sort and selection) kernels of a captured batch of n pairs."""
    b = CollisionBatch(st, n, graphs=False)
    with torch.cuda.stream(b.stream):
        b._launch(n)
    b.stream.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g, stream=b.stream):
        b._launch(n)
    own, toolkit = ctypes.c_int64(0), ctypes.c_int64(0)
    _lib.check(_lib.load().d3d_graph_kernel_nodes(ctypes.c_void_p(g.raw_cuda_graph()), ctypes.byref(own),
                                                  ctypes.byref(toolkit)))
    return toolkit.value


def test_sort_min_as_set(scene):
    st = scene[0]
    unsorted = sort_kernels(st, 8000)  # below a full grid: not sorted at the first setting
    set_tuning(sort_min=8000)
    assert sort_kernels(st, 8000) > unsorted
    assert sort_kernels(st, 7999) == unsorted
    set_tuning(sort_min=0)
    assert sort_kernels(st, 100) > unsorted
    set_tuning(sort_min=2 ** 31 - 1)
    full = 512 * torch.cuda.get_device_properties(0).multi_processor_count
    assert sort_kernels(st, full) == unsorted
    set_tuning(sort_min=4096)
    assert sort_kernels(st, full - 1) == unsorted
    assert sort_kernels(st, full) > unsorted


def test_unread_parameters_stay(scene):
    st, i1, i2 = scene
    for start in (dict(gjk_block=128, epa_warps=4), dict(gjk_block=64, epa_warps=8)):
        set_tuning(**start)
        sort_min = get_tuning()["sort_min"]
        for _ in range(3):
            t = autotune(st, i1, i2)
            # no sort below a full grid, and the phase's blocks hold 16 warps per SM at any size
            assert t["sort_min"] == sort_min and t["gjk_warps_per_sm"] == 0
            set_tuning(**start)
            t = autotune(st, i1, i2, precision="fp64")
            assert {k: t[k] for k in start} == start and t["gjk_warps_per_sm"] == 0
            set_tuning(sort_min=sort_min, **start)


@pytest.mark.parametrize("batches", [2, 6])
def test_batches(scene, batches):
    st, i1, i2 = scene
    n = 1500
    t = autotune(st, i1[:batches * n], i2[:batches * n], batches=batches)
    assert t == get_tuning()
    with pytest.raises(ValueError):
        autotune(st, i1[:batches * n - 1], i2[:batches * n - 1], batches=batches)
