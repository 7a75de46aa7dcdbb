"""The team kernel (one block per query, lists evaluated ahead) against the oracle: every distance at
row lengths on both sides of its 16- and 32-float blocks, lists on both sides of 32 and 64 ids, beams on
both sides of its block sizes, k above efSearch, SearchOld, equal distances everywhere, a table that
fills up, and NaN queries. Ids, distances and per-query counts must be identical."""
import struct

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


def _index(tmp_path, space, base, m, efc=64):
    path = str(tmp_path / "team.hnsw")
    lp = {"l1": 5, "linf": 6}.get(space)  # the builder has no L1 / LInf: an l2 graph under their distance code
    _capi.build_index(base, SPACES["l2" if lp else space], m, efc, nthreads=0, out_path=path)
    if lp:
        with open(path, "r+b") as f:
            f.seek(56)  # dist_func_type, after flag, counts, offsets, levels and maxM / maxM0
            f.write(struct.pack("<i", lp))
    idx = nmslib.init(method="hnsw", space=space)
    idx.loadIndex(path)
    return idx, OracleIndex(path)


def _check(idx, orc, q, k, ef, algo):
    idx.setQueryTimeParams({"efSearch": ef, "algoType": algo})
    ids, d, cnt, st = idx.knnQueryBatchArrays(q, k, stats=True)
    oi, od, oc, ost = orc.search(q, k=k, ef=ef, algo=ALGO_CODES[algo])
    np.testing.assert_array_equal(cnt, oc)
    np.testing.assert_array_equal(ids, oi)
    np.testing.assert_array_equal(d.view(np.int32), od.view(np.int32))
    np.testing.assert_array_equal(st, ost)


@pytest.mark.parametrize("space", ["l2", "cosinesimil", "negdotprod", "l1", "linf"])
@pytest.mark.parametrize("dim,m", [(5, 8), (16, 16), (33, 17), (47, 8), (100, 24), (112, 8), (128, 33), (159, 16)])
def test_shapes_and_beams(tmp_path, space, dim, m):
    rng = np.random.default_rng(dim * 100 + m)
    idx, orc = _index(tmp_path, space, rng.standard_normal((2000, dim)).astype(np.float32), m)
    q = rng.standard_normal((40, dim)).astype(np.float32)
    for k, ef in ((1, 1), (10, 64), (10, 65), (7, 128), (10, 257), (100, 40)):
        _check(idx, orc, q[:1 if ef == 64 else 40], k, ef, "v1merge")
    _check(idx, orc, q, 10, 50, "old")
    _check(idx, orc, q, 90, 50, "old")


@pytest.mark.parametrize("space", ["l2", "l1"])
def test_equal_distances(tmp_path, space):
    rng = np.random.default_rng(3)
    base = rng.integers(0, 3, (1500, 6)).astype(np.float32)  # few distinct rows: runs of equal distances
    idx, orc = _index(tmp_path, space, base, 16)
    q = rng.integers(0, 3, (64, 6)).astype(np.float32)
    for algo in ("v1merge", "old"):
        for k, ef in ((10, 20), (30, 90), (50, 200), (40, 15)):
            _check(idx, orc, q, k, ef, algo)


@pytest.mark.parametrize("algo", ["v1merge", "old"])
def test_table_that_fills_up(tmp_path, algo):
    """Enough queries that a block's table is its smallest, and a beam that visits most of the index."""
    rng = np.random.default_rng(5)
    idx, orc = _index(tmp_path, "l2", rng.standard_normal((9000, 24)).astype(np.float32), 16)
    _check(idx, orc, rng.standard_normal((700, 24)).astype(np.float32), 10, 1200, algo)


def test_nan_queries_stay_in_range(tmp_path):
    rng = np.random.default_rng(6)
    idx, _ = _index(tmp_path, "l2", rng.standard_normal((500, 20)).astype(np.float32), 8)
    q = np.full((3, 20), np.nan, np.float32)
    q[1, 3:] = 0.5
    q[2] = np.inf
    for algo in ("v1merge", "old"):
        idx.setQueryTimeParams({"efSearch": 30, "algoType": algo})
        ids, _, cnt = idx.knnQueryBatchArrays(q, 10)
        for r in range(3):
            got = ids[r, :cnt[r]]
            assert len(set(got.tolist())) == len(got) and (got >= 0).all() and (got < 500).all()
