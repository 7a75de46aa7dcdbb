"""Launch shapes that small automatic batches do not take, against the oracle: the team kernel with four
warps per block (more than eight queries per SM), its table of 2,048 entries filling up, its level-0 pass
behind a separate descent; and the lean kernel's single pass, with and without lists that repeat an id.
Ids, distances and per-query counts must be identical."""
import struct

import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import SPACES, _capi
from nmslib_b200.build import build
from oracle.oracle import OracleIndex

from conftest import ALGO_CODES, golden_path, load_golden

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build()


def _index(tmp_path, space, base, m):
    path = str(tmp_path / "shape.hnsw")
    lp = {"l1": 5, "linf": 6}.get(space)  # the builder has no L1 / LInf: an l2 graph under their distance code
    _capi.build_index(base, SPACES["l2" if lp else space], m, 32, nthreads=0, out_path=path)
    if lp:
        with open(path, "r+b") as f:
            f.seek(56)
            f.write(struct.pack("<i", lp))
    return _open(path, space)


def _open(path, space):
    idx = nmslib.init(method="hnsw", space=space)
    idx.loadIndex(path)
    return idx, OracleIndex(path)


def _check(idx, orc, q, k, ef, reps=1, **shape):
    idx.setQueryTimeParams({"efSearch": ef, "algoType": "v1merge"})
    idx.setLaunchConfig(**shape)
    ids, d, cnt, st = idx.knnQueryBatchArrays(np.tile(q, (reps, 1)), k, stats=True)
    oi, od, oc, ost = orc.search(q, k=k, ef=ef, algo=ALGO_CODES["v1merge"])
    np.testing.assert_array_equal(cnt, np.tile(oc, reps))
    np.testing.assert_array_equal(ids, np.tile(oi, (reps, 1)))
    np.testing.assert_array_equal(d.view(np.int32), np.tile(od, (reps, 1)).view(np.int32))
    np.testing.assert_array_equal(st, np.tile(ost, (reps, 1)))


@pytest.mark.parametrize("space,dim,nq", [(s, d, 1300) for s in ("l2", "cosinesimil", "negdotprod")
                                          for d in (27, 80, 112, 128, 159)] +
                         [("l1", 27, 1300), ("l1", 100, 2500), ("linf", 27, 1300), ("linf", 100, 2500)])
def test_four_warps(tmp_path, space, dim, nq):
    rng = np.random.default_rng(dim)
    idx, orc = _index(tmp_path, space, rng.standard_normal((6000, dim)).astype(np.float32), 16)
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    for k, ef in ((10, 128), (150, 100), (7, 300)):
        _check(idx, orc, q, k, ef)


@pytest.mark.parametrize("order", [0, -1], ids=["split", "one-pass"])
def test_four_warps_long_beams(tmp_path, order):
    """2,000 queries at efSearch 2000: more than the one-warp kernel holds, so level 0 is a pass of its own;
    a beam visits more ids than the table holds."""
    rng = np.random.default_rng(9)
    idx, orc = _index(tmp_path, "l2", rng.standard_normal((9000, 24)).astype(np.float32), 16)
    _check(idx, orc, rng.standard_normal((100, 24)).astype(np.float32), 10, 2000, reps=20, query_order=order)


@pytest.mark.parametrize("space", ["l2", "cosinesimil", "negdotprod"])
@pytest.mark.parametrize("dim,m", [(16, 24), (33, 8), (48, 8), (64, 24), (96, 16), (100, 24), (128, 32), (200, 8),
                                   (256, 24)])
def test_lean_single_pass(tmp_path, space, dim, m):
    rng = np.random.default_rng(dim + m)
    idx, orc = _index(tmp_path, space, rng.standard_normal((2000, dim)).astype(np.float32), m)
    q = rng.standard_normal((300, dim)).astype(np.float32)
    for k, ef in ((10, 10), (10, 64), (100, 40), (10, 300)):
        _check(idx, orc, q, k, ef, warps_per_block=4)


@pytest.mark.parametrize("shape", [dict(), dict(warps_per_block=4)], ids=["team", "lean"])
def test_lists_that_repeat_an_id(tmp_path, shape):
    raw = bytearray(open(golden_path("c1_l2_d128"), "rb").read())
    n, mem, off0 = struct.unpack_from("<IQQ", raw, 4)
    for i in range(0, n, 3):
        p = 68 + i * mem + off0
        if struct.unpack_from("<i", raw, p)[0] >= 3:
            raw[p + 12:p + 16] = raw[p + 4:p + 8]  # the third id is the first again
    path = tmp_path / "repeated.hnsw"
    path.write_bytes(bytes(raw))
    idx, orc = _open(str(path), "l2")
    for ef in (10, 64, 300):
        _check(idx, orc, load_golden("c1_l2_d128")["queries"], 10, ef, **shape)
