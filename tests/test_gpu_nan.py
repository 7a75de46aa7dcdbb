"""NaN distances (an infinite query coordinate against rows with zeros there, NaN rows, NaN queries) in every
search kernel. A NaN distance counts as infinite; every result is a row of the index, once, in ascending
order."""
import struct

import numpy as np
import pytest

import nmslib_b200 as nmslib
from nmslib_b200 import SPACES, _capi
from nmslib_b200.build import build

pytestmark = pytest.mark.gpu
N = 2000


def _index(path, space, dim, nan_rows):
    """Sparse rows; `nan_rows`: the entry point and every 50th row get a NaN after the graph is built."""
    rng = np.random.default_rng(dim)
    base = rng.standard_normal((N, dim)).astype(np.float32)
    base[rng.random(base.shape) < 0.5] = 0.0
    lp = {"l1": 5, "linf": 6}.get(space)
    _capi.build_index(base, SPACES["l2" if lp else space], 16, 64, nthreads=0, out_path=path)
    raw = bytearray(open(path, "rb").read())
    if lp:
        struct.pack_into("<i", raw, 56, lp)
    if nan_rows:
        mem, entry = struct.unpack_from("<Q", raw, 8)[0], struct.unpack_from("<i", raw, 36)[0]
        for row in (entry, *range(0, N, 50)):
            struct.pack_into("<f", raw, 68 + row * mem + 16, float("nan"))
    with open(path, "wb") as f:
        f.write(raw)
    idx = nmslib.init(method="hnsw", space=space)
    idx.loadIndex(path)
    return idx, rng


SHAPES = [({}, 96), ({}, 1300), ({}, 7000), (dict(warps_per_block=4), 96), (dict(rows_per_group=1, stage_rows=-1), 96),
          (dict(queries_per_warp=2), 96), (dict(visited_hash_log2=10), 96)]


@pytest.mark.parametrize("nan_rows", [False, True])
@pytest.mark.parametrize("space,dim", [("negdotprod", 96), ("negdotprod", 100), ("l2", 48), ("cosinesimil", 100),
                                       ("l1", 40), ("linf", 40)])
def test_nan_distances_stay_in_range(tmp_path, space, dim, nan_rows):
    build()
    idx, rng = _index(str(tmp_path / "nan.hnsw"), space, dim, nan_rows)
    q = rng.standard_normal((7000, dim)).astype(np.float32)
    q[0::4, 3] = np.inf
    q[1::4, 5] = -np.inf
    q[2::16] = np.nan
    for shape, nq in SHAPES:
        for algo, k, ef in (("v1merge", 10, 30), ("v1merge", 10, 200), ("v1merge", 40, 20), ("old", 10, 100)):
            idx.setQueryTimeParams({"efSearch": ef, "algoType": algo})
            idx.setLaunchConfig(**shape)
            ids, d, cnt = idx.knnQueryBatchArrays(q[:nq], k)
            assert (d[:, 1:] >= d[:, :-1]).all()
            assert (cnt >= 1).all() and (cnt <= k).all()
            live = np.arange(k) < cnt[:, None]
            assert (ids[live] >= 0).all() and (ids[live] < N).all() and (ids[~live] == -1).all()
            s = np.sort(np.where(live, ids, -1 - np.arange(k)), axis=1)
            assert (s[:, 1:] != s[:, :-1]).all()
