"""Host arrays on both sides of 512 KB (staging and direct copies) and 1 MB (a call's block), page-locked
and pageable, queries and results apart: searches and exact scans return the same bytes."""
import ctypes

import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import _capi
from nmslib_b200.build import build

from conftest import golden_path, load_golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def index():
    build()
    idx = nmslib.init(method="hnsw", space="l2")
    idx.loadIndex(golden_path("c1_l2_d128"))
    idx.setQueryTimeParams({"efSearch": 64, "algoType": "v1merge"})
    return idx


@pytest.mark.parametrize("call", ["search", "exact"])
@pytest.mark.parametrize("nq,k", [(900, 10), (1100, 32), (2100, 32), (4500, 32)])
def test_same_results_from_any_host_memory(index, call, nq, k):
    import torch

    q0 = np.resize(load_golden("c1_l2_d128")["queries"], (nq, 128))
    lib = _capi.load()
    want = None
    for locked_q in (False, True):
        for locked_r in (False, True):
            q = torch.from_numpy(q0).clone()
            q = q.pin_memory() if locked_q else q
            out = [torch.full(s, -3, dtype=t, pin_memory=locked_r)
                   for s, t in (((nq, k), torch.int32), ((nq, k), torch.float32), ((nq,), torch.int32))]
            p = [ctypes.c_void_p(t.data_ptr()) for t in (q, *out)]
            if call == "search":
                rc = lib.nmsg_knn_batch(index._require(), p[0], nq, 128, k, None, None, k, *p[1:], None, 0, None)
            else:
                rc = lib.nmsg_bruteforce_knn(index._require(), p[0], nq, 128, k, k, *p[1:], None, 0, None)
            _capi.check(rc)
            got = [t.numpy().copy() for t in out]
            if want is None:
                want = got
                assert (got[2] == k).all()
            for x, y in zip(got, want):
                np.testing.assert_array_equal(x.view(np.int32), y.view(np.int32))
