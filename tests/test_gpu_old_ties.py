"""SearchOld where a few rows are equal among distinct ones, so that the walk's own result is kept instead
of the heaps': a result queue that holds k rejects an equal distance, so of equal rows at the k-th place
the one found first stays. Ids, distances and per-query counts must be the oracle's."""
import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import SPACES, _capi
from nmslib_b200.build import build
from oracle.oracle import OracleIndex

from conftest import ALGO_CODES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build()


def _open(path):
    idx = nmslib.init(method="hnsw", space="l2")
    idx.loadIndex(path)
    return idx, OracleIndex(path)


def _check(idx, orc, q, k, ef, algo):
    idx.setQueryTimeParams({"efSearch": ef, "algoType": algo})
    ids, d, cnt, st = idx.knnQueryBatchArrays(q, k, stats=True)
    oi, od, oc, ost = orc.search(q, k=k, ef=ef, algo=ALGO_CODES[algo])
    np.testing.assert_array_equal(cnt, oc)
    np.testing.assert_array_equal(d.view(np.int32), od.view(np.int32))
    np.testing.assert_array_equal(ids, oi)
    np.testing.assert_array_equal(st, ost)


@pytest.fixture(scope="module")
def pairs(tmp_path_factory):
    """20,000 continuous rows, 6,000 of them in equal pairs, and queries near the paired rows."""
    rng = np.random.default_rng(41)
    base = rng.standard_normal((20000, 16)).astype(np.float32)
    base[3000:6000] = base[:3000]
    base = base[rng.permutation(len(base))]
    path = str(tmp_path_factory.mktemp("old_ties") / "pairs.hnsw")
    _capi.build_index(base, SPACES["l2"], 16, 100, nthreads=0, out_path=path)
    q = base[rng.integers(0, len(base), 2400)] + 0.05 * rng.standard_normal((2400, 16))
    return *_open(path), q.astype(np.float32)


@pytest.mark.parametrize("k", [1, 2, 3, 10])
@pytest.mark.parametrize("ef,algo", [(200, "old"), (1000, "hybrid")])
def test_equal_rows_at_the_last_place(pairs, ef, algo, k):
    _check(*pairs, k, ef, algo)
