"""SearchOld where a few rows are equal among distinct ones, so that the walk's own result is kept instead
of the heaps': a result queue that holds k rejects an equal distance, so of equal rows at the k-th place
the one found first stays. Also a run of expansions that keeps more neighbours than a block has threads
and leaves one of two equal candidates at the array's end. Ids, distances and per-query counts must be
the oracle's."""
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


def _write_l2(path, rows, lists, m):
    """A one-level optimized index of the reference's layout: header, packed rows, no upper lists."""
    n, dim = rows.shape
    row = np.zeros((n, 4 + dim + 1 + 2 * m), np.int32)
    row[:, 0] = np.arange(n)
    row[:, 1] = -1
    row[:, 2] = 4 * dim
    row[:, 4:4 + dim] = rows.view(np.int32)
    for i, lst in lists.items():
        row[i, 4 + dim] = len(lst)
        row[i, 5 + dim:5 + dim + len(lst)] = lst
    with open(path, "wb") as f:
        f.write(np.array([1, n], np.uint32).tobytes())
        f.write(np.array([4 * row.shape[1], 16 + 4 * dim, 0], np.uint64).tobytes())
        f.write(np.array([0, 0], np.int32).tobytes())
        f.write(np.array([m, 2 * m], np.uint64).tobytes())
        f.write(np.int32(1).tobytes() + np.uint64(3).tobytes())
        f.write(row.tobytes())
        f.write(np.zeros(n, np.uint32).tobytes())


@pytest.mark.parametrize("leads", [0, 1])
def test_equal_candidates_cut_apart_by_a_long_run(tmp_path, leads):
    """The entry names 16 near rows and two equal far ones. The near rows' lists then bring 768
    neighbours in one run, 283 of them nearer than the equal pair: of 300 places the last is one of the
    pair's, and SearchOld still expands both. One of them leads to the nearest row of all."""
    near, pair, first = range(1, 17), (17, 18), 19
    mid = np.concatenate([np.arange(17, 300), np.arange(501, 501 + 768 - 283)]).astype(np.float32)
    mid = mid[np.random.default_rng(2).permutation(768)]
    rows = np.zeros((first + 769, 16), np.float32)
    rows[0, 0] = 2000
    rows[list(near), 0] = list(near)
    rows[list(pair), 0] = 500
    rows[first:first + 768, 0] = mid
    rows[first + 768, 0] = 0.5
    lists = {0: [*near, *pair], pair[leads]: [first + 768]}
    for i in range(8):
        lists[1 + i] = list(range(first + 96 * i, first + 96 * (i + 1)))
    path = str(tmp_path / "apart.hnsw")
    _write_l2(path, rows, lists, 48)
    idx, orc = _open(path)
    q = np.zeros((1, 16), np.float32)
    assert orc.search(q, k=10, ef=300, algo=ALGO_CODES["old"])[0][0, 0] == first + 768
    _check(idx, orc, q, 10, 300, "old")
