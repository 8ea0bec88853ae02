"""Sizes at the edges of the scan kernels' tiles, on the GPU: base tiles, query tiles, K
chunks and the selection regimes of the tensor-core scans, each against the general path
or the CPU oracle.  Sketch distances are integers and distances are the reference's
single-precision formula on both sides, so everything is compared for equality.
"""
import numpy as np
import pytest

from lshongpu_gb300 import datasets

pytestmark = pytest.mark.gpu

D = 100
POPCOUNT, TENSOR = 1, 2


def data(n, nq, d=D, seed=61, count=40):
    return datasets.clustered(n, d, seed, count=count), datasets.clustered(nq, d, seed + 1, count=count)


@pytest.mark.parametrize("n,nq,words,C", [
    (224, 1, 1, 32),          # one full base tile, one query, one K step
    (225, 128, 2, 32),        # one point in the second tile
    (16352, 129, 8, 256),     # the largest base that keeps every point; a query tile of one row
    (16353, 257, 9, 256),     # one more: prepass; a cluster with one query tile; a second chunk of one word
    (50176, 384, 17, 512),    # whole tiles; 3 query tiles; 3 chunks
    (140001, 100, 25, 4096),  # 4 chunks (the last of one word), 8-point groups, one query tile
])
def test_sketch_scan_edges_equal_popcount(engine, n, nq, words, C):
    """The FP4 sketch scan (base tiles of 224 points, clusters of two 128-row query tiles,
    chunks of 8 words) returns what the popcount scan returns."""
    x, q = data(n, nq)
    res = [engine.Index(x, implementation=3, sketchDim=words,
                        options=engine.make_options(candidates=C, sketch_scan=mode)).query(q, 32)
           for mode in (TENSOR, POPCOUNT)]
    assert np.array_equal(res[0], res[1])


@pytest.mark.parametrize("n,nq,k,d", [
    (256 * 64, 1, 10, 64),       # whole tiles, one K chunk, one query
    (256 * 64 + 1, 128, 32, 65),  # one point in the last tile; a second chunk of one K step
    (70000, 129, 32, 100),       # a query tile of one row: a cluster's second CTA
    (70000, 257, 100, 37),       # three query tiles in two clusters; 128 candidates
    (40001, 900, 32, 128),       # eight query tiles: clusters keep theirs
    (40001, 1300, 32, 16),       # eleven: clusters change theirs; one K step
])
@pytest.mark.parametrize("impl", [8, 9])
def test_filter_scan_edges_equal_list_kernel(engine, monkeypatch, n, nq, k, d, impl):
    """The tensor-core filter scan selects what the exact per-row list kernel selects from
    the same BF16 scores.  With E4M3 scores (the list kernel has BF16 ones only): a row of the
    batch equals its own query, and every distance is the exact scan's for that id."""
    x, q = data(n, nq, d)
    idx = engine.Index(x, implementation=impl, distanceFunc=1)
    res = idx.query(q, k)
    if impl == 8:
        monkeypatch.setenv("LSHG_TC_FORCE_FALLBACK", "1")
        assert np.array_equal(res, idx.query(q, k))
        return
    assert np.array_equal(res[:1], idx.query(q[:1], k))
    ex = engine.Index(x, implementation=2, distanceFunc=1).query(q, k)
    for a, b in zip(res, ex):
        exact = dict(zip(b["ID"].tolist(), b["distance"].tolist()))
        assert len(set(a["ID"].tolist())) == k
        for i, dist in zip(a["ID"].tolist(), a["distance"].tolist()):
            assert exact.get(i, dist) == dist
