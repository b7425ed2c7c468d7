"""A server of many slots launches its batches for a shared GPU (few full
blocks); the results are those of a batch that has the GPU to itself."""
import numpy as np
import pytest

from distance3d_gb300 import workloads
from distance3d_gb300.serve import CollisionBatch, NativeCollisionServer
from distance3d_gb300.store import ColliderStore

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("faces,edges", [(64, 32), (256, 128)])
def test_many_slots(graphs, precision, faces, edges):
    cs, i1, i2 = workloads.pairs_mixed_six(9000, seed=4, center_half_width=0.38)
    st = ColliderStore(cs)
    i1, i2 = np.asarray(i1, np.int32), np.asarray(i2, np.int32)
    kw = dict(max_iter=64, max_loose_edges=edges, max_faces=faces, epsilon=1e-8)
    ref = CollisionBatch(st, 16384, precision=precision, epa_kw=kw, graphs=False)
    srv = NativeCollisionServer(st, capacity=4096, slots=6, precision=precision, epa_kw=kw, graphs=graphs)
    try:
        cuts = [(0, 1), (1, 32), (32, 161), (161, 4257), (4257, 9000)]
        tickets = [srv.submit(i1[a:b], i2[a:b]) for a, b in cuts]
        for (a, b), t in zip(cuts, tickets):
            out, _ = srv.result(t)
            alone = ref.run(i1[a:b], i2[a:b])
            for k in alone:
                assert np.array_equal(out[k], alone[k], equal_nan=True), (a, b, k)
    finally:
        srv.close()
