"""The exact rerank of the tensor-core brute force where a query has more candidates than the kernel
holds in shared memory (2,048), or more rows with exact keys than its buffer (512), against a float64
scan: few distinct rows, so that whole classes of them tie and the smallest ids win."""
import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import SPACES, _capi
from nmslib_b200.build import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space", ["l2", "negdotprod"])
@pytest.mark.parametrize("n,distinct,nq,k", [(600, 1, 1, 32), (3000, 1, 2, 1), (12000, 3, 3, 32), (12000, 40, 130, 7)])
def test_many_tied_candidates(tmp_path, space, n, distinct, nq, k):
    build()
    rng = np.random.default_rng(n + distinct)
    rows = rng.integers(-3, 4, (distinct, 24)).astype(np.float32)
    base = rows[rng.integers(0, distinct, n)]
    path = str(tmp_path / "ties.hnsw")
    _capi.build_index(base, SPACES[space], 4, 8, nthreads=0, out_path=path)
    idx = nmslib.init(method="hnsw", space=space)
    idx.loadIndex(path)
    q = rng.integers(-3, 4, (nq, 24)).astype(np.float32)
    ids, d, cnt = idx.bruteForceBatchArrays(q, k)
    dot = q.astype(np.float64) @ base.T.astype(np.float64)
    want = -dot if space == "negdotprod" else (q ** 2).sum(1)[:, None] + (base ** 2).sum(1) - 2 * dot
    order = np.argsort(want, axis=1, kind="stable")[:, :k]  # equal distances by id
    np.testing.assert_array_equal(cnt, np.full(nq, k))
    np.testing.assert_array_equal(ids, order)
    np.testing.assert_array_equal(d, np.take_along_axis(want, order, 1).astype(np.float32))
