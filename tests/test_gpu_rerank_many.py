"""The exact rerank's shapes for many queries (128 threads past four queries per SM, 64 past sixteen for short
results): more candidates than they hold in shared memory (1,024 and 512), more rows with exact keys than
their buffers (288 and 160), and ordinary rows, against a float64 scan."""
import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import SPACES, _capi
from nmslib_b200.build import build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space", ["l2", "negdotprod"])
@pytest.mark.parametrize("n,distinct,nq,k", [(200, 1, 700, 32), (900, 1, 700, 1), (12000, 3, 700, 32), (9000, 9000, 700, 32),
                                             (200, 1, 2500, 16), (3000, 1, 2500, 1), (12000, 3, 2500, 16),
                                             (9000, 40, 2500, 7), (9000, 9000, 2500, 10), (3000, 2, 2500, 17)])
def test_many_queries(tmp_path, space, n, distinct, nq, k):
    build()
    rng = np.random.default_rng(n + distinct + nq)
    rows = rng.integers(-30, 31, (distinct, 24)).astype(np.float32)
    base = rows[rng.integers(0, distinct, n)] if distinct < n else rows
    path = str(tmp_path / "many.hnsw")
    _capi.build_index(base, SPACES[space], 4, 8, nthreads=0, out_path=path)
    idx = nmslib.init(method="hnsw", space=space)
    idx.loadIndex(path)
    q = rng.integers(-30, 31, (nq, 24)).astype(np.float32)
    ids, d, cnt = idx.bruteForceBatchArrays(q, k)
    dot = q.astype(np.float64) @ base.T.astype(np.float64)
    want = -dot if space == "negdotprod" else (q ** 2).sum(1)[:, None] + (base ** 2).sum(1) - 2 * dot
    order = np.argsort(want, axis=1, kind="stable")[:, :k]  # equal distances by id
    np.testing.assert_array_equal(cnt, np.full(nq, k))
    np.testing.assert_array_equal(ids, order)
    np.testing.assert_array_equal(d, np.take_along_axis(want, order, 1).astype(np.float32))
