"""Small batches side by side on several streams: each gives the results it
gives alone, and they share the GPU instead of running one after the other."""
import time

import numpy as np
import pytest
import torch

from distance3d_gb300 import workloads
from distance3d_gb300.gjk import gjk_distance_batch, gjk_intersection_batch
from distance3d_gb300.mpr import mpr_batch
from distance3d_gb300.store import ColliderStore

pytestmark = pytest.mark.gpu

STREAMS = 16


def _batches(n):
    cs, i1, i2 = workloads.pairs_mixed_six(STREAMS * n, seed=11, center_half_width=0.38)
    st = ColliderStore(cs)
    t = [torch.as_tensor(np.asarray(x, np.int32), device=st.device) for x in (i1, i2)]
    return st, [(t[0][k * n:(k + 1) * n], t[1][k * n:(k + 1) * n]) for k in range(STREAMS)]


def _side_by_side(call, reps=1):
    streams = [torch.cuda.Stream() for _ in range(STREAMS)]
    torch.cuda.synchronize()
    out = [None] * STREAMS
    for _ in range(reps):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                out[k] = call(k)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("n", [33, 1000, 4097])
@pytest.mark.parametrize("form", ["fp64", "mixed", "hit", "mpr"])
def test_same_results(form, n):
    st, p = _batches(n)
    call = {"fp64": lambda k: gjk_distance_batch(st, *p[k]),
            "mixed": lambda k: gjk_distance_batch(st, *p[k], precision="mixed"),
            "hit": lambda k: gjk_intersection_batch(st, *p[k]),
            "mpr": lambda k: mpr_batch(st, *p[k])}[form]
    alone = []
    for k in range(STREAMS):
        alone.append(call(k))
        torch.cuda.synchronize()
    for a, b in zip(alone, _side_by_side(call, reps=3)):
        for key in a:
            assert np.array_equal(a[key].cpu().numpy(), b[key].cpu().numpy(), equal_nan=True), (form, n, key)


def test_batches_share_the_gpu():
    # 4,000 pairs fill 16 of the FP64 pool's 304 resident blocks, so 16 batches fit at once; with the
    # pairs packed that densely a batch's own chain is about twice as long, which leaves a factor of
    # ~7 over one batch after the other.  A third of it is asked for.
    n = 4000
    st, p = _batches(n)
    out = [gjk_distance_batch(st, *p[k]) for k in range(STREAMS)]

    def call(k):
        return gjk_distance_batch(st, *p[k], out=out[k])

    def seconds(run):
        best = 1e9
        for _ in range(4):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            run()
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        return best

    serial = seconds(lambda: [call(k) for _ in range(4) for k in range(STREAMS)])
    beside = seconds(lambda: _side_by_side(call, reps=4))
    assert serial / beside > 2.3, (serial, beside)
