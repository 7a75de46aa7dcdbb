"""The lean kernel for rows with a remainder past a multiple of 16 floats, against the oracle: every
instantiated length class with remainders of 1 to 15, lists of up to 32 and up to 64 ids, batches that
are split (descent pass, order, level-0 pass) and that are not. Ids, distances and per-query counts must
be identical."""
import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import SPACES, _capi
from nmslib_b200.build import build
from oracle.oracle import OracleIndex

from conftest import ALGO_CODES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space", ["l2", "cosinesimil", "negdotprod"])
@pytest.mark.parametrize("dim,m", [(33, 8), (52, 24), (67, 16), (95, 8), (100, 24), (105, 8), (127, 16), (130, 32),
                                   (200, 8), (201, 24)])
def test_rows_with_a_remainder(tmp_path, space, dim, m):
    build()
    rng = np.random.default_rng(dim * 100 + m)
    base = rng.standard_normal((2000, dim)).astype(np.float32)
    q = rng.standard_normal((250, dim)).astype(np.float32)
    path = str(tmp_path / "tail.hnsw")
    _capi.build_index(base, SPACES[space], m, 48, nthreads=0, out_path=path)
    idx = nmslib.init(method="hnsw", space=space)
    idx.loadIndex(path)
    orc = OracleIndex(path)
    for ef, k, reps in ((64, 10, 40), (200, 10, 20), (40, 60, 14)):
        idx.setQueryTimeParams({"efSearch": ef, "algoType": "v1merge"})
        ids, d, cnt, st = idx.knnQueryBatchArrays(np.tile(q, (reps, 1)), k, stats=True)
        oi, od, oc, ost = orc.search(q, k=k, ef=ef, algo=ALGO_CODES["v1merge"])
        np.testing.assert_array_equal(cnt, np.tile(oc, reps))
        np.testing.assert_array_equal(ids, np.tile(oi, (reps, 1)))
        np.testing.assert_array_equal(d.view(np.int32), np.tile(od, (reps, 1)).view(np.int32))
        np.testing.assert_array_equal(st, np.tile(ost, (reps, 1)))
