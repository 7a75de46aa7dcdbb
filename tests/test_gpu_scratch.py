"""Search scratch that grows or is new while calls run on a stream of the caller's: device-buffer batches
of growing size and beam on a non-blocking stream, and batches captured after a call with one query has
sized the scratch. Ids, distances and counts must be the oracle's."""
import ctypes

import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import _capi
from nmslib_b200.build import build
from oracle.oracle import OracleIndex

from conftest import golden_path, load_golden

pytestmark = pytest.mark.gpu
NAME = "c1_l2_d128"


class _Batch:
    def __init__(self, idx, nq, k):
        import torch

        self.rows = np.arange(nq) % 1000
        self.idx, self.k = idx, k
        self.q = torch.from_numpy(load_golden(NAME)["queries"][self.rows]).cuda()
        self.ids = torch.full((nq, k), -7, dtype=torch.int32, device="cuda")
        self.d = torch.zeros((nq, k), device="cuda")
        self.c = torch.zeros(nq, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

    def launch(self, stream):
        p = [ctypes.c_void_p(t.data_ptr()) for t in (self.q, self.ids, self.d, self.c)]
        _capi.check(_capi.load().nmsg_knn_batch(self.idx._require(), p[0], *self.q.shape, self.k, None, None, self.k,
                                                *p[1:], None, _capi.FLAG_DEVICE_PTRS,
                                                ctypes.c_void_p(stream.cuda_stream)))

    def check(self, want):
        oi, od, oc, _ = want
        np.testing.assert_array_equal(self.c.cpu().numpy(), oc[self.rows])
        np.testing.assert_array_equal(self.ids.cpu().numpy(), oi[self.rows])
        np.testing.assert_array_equal(self.d.cpu().numpy().view(np.int32), od[self.rows].view(np.int32))


def _index():
    build()
    idx = nmslib.init(method="hnsw", space="l2")
    idx.loadIndex(golden_path(NAME))
    return idx, OracleIndex(golden_path(NAME))


@pytest.mark.parametrize("efs", [(64,), (400, 64, 16)], ids=["batch", "batch-and-beam"])
def test_growing_batches_on_a_non_blocking_stream(efs):
    import torch

    idx, orc = _index()
    q = load_golden(NAME)["queries"]
    stream = torch.cuda.Stream()  # made non-blocking
    for ef in efs:
        idx.setQueryTimeParams({"efSearch": ef, "algoType": "v1merge"})
        want = orc.search(q, k=10, ef=ef, algo=2)
        batches = [_Batch(idx, nq, 10) for nq in (1, 300, 1300, 2500, 7000)]
        for b in batches:
            b.launch(stream)
        stream.synchronize()
        for b in batches:
            b.check(want)


@pytest.mark.parametrize("nq", [300, 1300, 2300])
def test_capture_after_a_small_call(nq):
    import torch

    idx, orc = _index()
    idx.setQueryTimeParams({"efSearch": 64, "algoType": "v1merge"})
    stream = torch.cuda.Stream()
    one, many = _Batch(idx, 1, 10), _Batch(idx, nq, 10)
    one.launch(stream)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        many.launch(stream)
    graph.replay()
    torch.cuda.synchronize()
    many.check(orc.search(load_golden(NAME)["queries"], k=10, ef=64, algo=2))
