"""d3d_gjk_intersection takes no memory but its arguments: a captured call is
one kernel node (no allocation or memory nodes), which replays beside itself,
and its pairs are dealt to the blocks in input order at any batch size."""
import ctypes

import numpy as np
import pytest
import torch

from distance3d_gb300 import _lib, workloads
from distance3d_gb300.gjk import gjk_intersection_batch
from distance3d_gb300.store import ColliderStore, _ptr
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_block", [0, 1, 31, 255, 256, 257, 300])
def test_captured_call_is_one_kernel(per_block):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = per_block * 2 * sms + 7  # two blocks of 256 pairs are resident per SM
    cs, i1, i2 = workloads.pairs_all_types(n, seed=n, margin_fraction=0.2)
    st = ColliderStore(cs)
    a, b = (torch.as_tensor(np.asarray(x, np.int32), device=st.device) for x in (i1, i2))
    hit = torch.full((n,), -1, dtype=torch.int8, device=st.device)
    status = torch.full((n,), -1, dtype=torch.int8, device=st.device)
    stream = torch.cuda.Stream()

    def call():
        _lib.check(_lib.load().d3d_gjk_intersection(st.view, _ptr(a), _ptr(b), n, 1e-10, 1024, _ptr(hit), _ptr(status),
                                                    ctypes.c_void_p(stream.cuda_stream)))

    call()
    stream.synchronize()
    ref = oracle.gjk_intersection(cs, i1, i2)
    assert np.array_equal(hit.cpu().numpy().astype(bool), ref["hit"])
    assert np.array_equal(status.cpu().numpy(), ref["status"])
    hit.fill_(-1)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g, stream=stream):
        call()
    nodes = ctypes.c_size_t(0)
    cuda = ctypes.CDLL("libcuda.so.1")
    assert cuda.cuGraphGetNodes(ctypes.c_void_p(g.raw_cuda_graph()), None, ctypes.byref(nodes)) == 0
    assert nodes.value == 1
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(hit.cpu().numpy().astype(bool), ref["hit"])


def test_out_of_range_pairs_among_others():
    n = 5000
    cs, i1, i2 = workloads.pairs_all_types(n, seed=3)
    i1, i2 = np.array(i1, np.int32), np.array(i2, np.int32)
    ref = oracle.gjk_intersection(cs, i1, i2)
    bad = np.arange(0, n, 7)
    i1[bad[::2]] = -1
    i2[bad[1::2]] = len(cs)
    st = ColliderStore(cs)
    a, b = (torch.as_tensor(x, device=st.device) for x in (i1, i2))
    r = gjk_intersection_batch(st, a, b)
    status = r["status"].cpu().numpy()
    assert (status[bad] == _lib.STATUS_BAD_INDEX).all() and not r["hit"].cpu().numpy()[bad].any()
    good = np.setdiff1d(np.arange(n), bad)
    assert np.array_equal(r["hit"].cpu().numpy()[good], ref["hit"][good])
