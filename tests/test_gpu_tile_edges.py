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


def scan_fp32(engine, idx, q, k):
    """The FP32 scan of an exact index (the allocation-free entry point runs nothing else)."""
    import torch

    dq = torch.from_numpy(q).cuda()
    out = torch.empty((q.shape[0], k, 2), dtype=torch.int32, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert engine.lib().lshg_index_query_noalloc(idx.handle, dq.data_ptr(), q.shape[0], k, out.data_ptr(),
                                                 st.cuda_stream) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy().view(engine.POINT_DTYPE).reshape(q.shape[0], k)


@pytest.mark.parametrize("n,nq,k,d", [
    (4096, 1, 1, 16),        # the smallest filtered base; one K step; one neighbour
    (4097, 129, 32, 64),     # one point in the last tile; a query tile of one row
    (20011, 257, 33, 65),    # 256 candidates; a second K chunk of one step
    (70000, 300, 128, 100),  # the largest filtered k
    (70000, 300, 10, 127),   # rows that are not 16-byte multiples
    (300000, 700, 32, 100),  # a sampled prepass
    (5000, 40, 200, 100),    # k beyond the filter: the FP32 scan
    (5000, 40, 32, 129),     # d beyond it
])
def test_exact_filter_equals_fp32_scan(engine, monkeypatch, n, nq, k, d):
    """Ids and distances of the filtered exact scan, and of its listed form, are the FP32
    scan's bit for bit; queries with no direction, no finite norm or a norm out of range
    included, and scaled queries (angular distance does not see the scale, FP32 rounding does)."""
    x, q = data(n, nq, d)
    q[::7] *= np.float32(1000.3)
    q[1::11] *= np.float32(1e-9)
    if nq > 20:
        q[3] = 0
        q[5, 0] = np.nan
        q[7, d - 1] = np.inf
        q[9] *= np.float32(1e18)
        q[11] *= np.float32(1e-25)
        q[13] = x[n - 1]
    idx = engine.Index(x, implementation=2, distanceFunc=1)
    want = scan_fp32(engine, idx, q, k)
    assert idx.query(q, k).tobytes() == want.tobytes()
    monkeypatch.setenv("LSHG_TC_FORCE_FALLBACK", "1")
    assert idx.query(q, k).tobytes() == want.tobytes()


@pytest.mark.parametrize("case", ["duplicates", "near ties", "zero row", "nan row", "huge row", "isotropic"])
def test_exact_filter_hard_bases(engine, case):
    """Bases that leave the filter too many candidates, or none of its bounds, give the FP32
    scan's results too."""
    n, d, nq, k = 30000, 100, 150, 32
    x, q = data(n, nq, d)
    if case == "duplicates":
        x[::2] = x[0]
        q[:50] = x[0]
    elif case == "near ties":  # every point within the scores' error of every other
        rng = np.random.default_rng(3)
        x = (x[:1] + 1e-4 * rng.standard_normal((n, d))).astype(np.float32)
    elif case == "isotropic":
        rng = np.random.default_rng(4)
        x, q = rng.standard_normal((n, d)).astype(np.float32), rng.standard_normal((nq, d)).astype(np.float32)
    else:
        x[12345] = {"zero row": 0.0, "nan row": np.nan, "huge row": 1e17}[case]
    idx = engine.Index(x, implementation=2, distanceFunc=1)
    assert idx.query(q, k).tobytes() == scan_fp32(engine, idx, q, k).tobytes()


def test_exact_filter_saved_index(engine, tmp_path):
    """A loaded exact index derives the filter's rows again; its file does not hold them."""
    x, q = data(9000, 200)
    idx = engine.Index(x, implementation=2, distanceFunc=1)
    path = str(tmp_path / "exact.lshg")
    idx.save(path)
    assert (tmp_path / "exact.lshg").stat().st_size < 9000 * 100 * 4 * 2.2
    assert engine.Index.load(path).query(q, 32).tobytes() == idx.query(q, 32).tobytes()


@pytest.mark.parametrize("impl", [4, 10])
@pytest.mark.parametrize("n,nq,S,C", [
    (10000, 1, 256, 128),    # one query; candidates by the warp select
    (4700, 3, 64, 1024),     # the sample barely holds the rank
    (17000, 65, 96, 4096),   # a second block of queries; candidates a quarter of the base
    (129, 2, 32, 32),        # one point in the second tile
])
def test_sample_filter_edges_equal_direct(engine, impl, n, nq, S, C):
    """Small batches, short lists and small bases of byte MinHash (4) and consistent weighted
    samples (10): the threshold filter's results are the direct scan's."""
    x, q = datasets.sparse_gamma(n, D, 71), datasets.sparse_gamma(nq, D, 72)
    res = [engine.Index(x, implementation=impl, distanceFunc=2, sketchDim=S,
                        options=engine.make_options(candidates=C, sketch_scan=mode)).query(q, 32)
           for mode in (0, TENSOR, POPCOUNT)]
    assert np.array_equal(res[0], res[2])
    assert np.array_equal(res[1], res[2])


@pytest.mark.parametrize("n,nq,words,C", [
    (10000, 1, 4, 128),      # below the pairs that take the tensor cores
    (36800, 2, 8, 4096),     # the largest base that keeps every point at C = 4,096
    (37000, 3, 8, 4096),     # 8-point maxima of every tile, rank near their number
    (20000, 5, 32, 2048),
])
def test_sketch_scan_small_batches_equal_popcount(engine, n, nq, words, C):
    x, q = data(n, nq)
    res = [engine.Index(x, implementation=3, sketchDim=words,
                        options=engine.make_options(candidates=C, sketch_scan=mode)).query(q, 32)
           for mode in (0, TENSOR, POPCOUNT)]
    assert np.array_equal(res[0], res[2])
    assert np.array_equal(res[1], res[2])


@pytest.mark.parametrize("n,nq,k,d,dist", [
    (500, 3, 32, 100, 2),     # one split
    (5000, 70, 64, 37, 2),    # lists of 64, rows with an odd pitch
    (60013, 129, 100, 64, 3),  # many splits, lists of 128
    (3000, 5, 300, 65, 2),    # lists beyond the short merge
    (70000, 2, 10, 130, 1),   # an FP32 angular scan of many splits
])
def test_exact_scan_split_merges(engine, orc, n, nq, k, d, dist):
    """The FP32 scan's split lists merge to the oracle's top-k: ids and distances of the Jaccard
    and angular scans bit for bit; Euclidean distances within the two square's rounding of
    the oracle's (d terms, 2^-24 each), in order."""
    if dist == 2:
        x, q = datasets.sparse_gamma(n, d, 91), datasets.sparse_gamma(nq, d, 92)
        xo, qo = orc.normalize(x), orc.normalize(q)
    else:
        x, q = data(n, nq, d)
        xo, qo = x, q
    res = engine.Index(x, implementation=2, distanceFunc=dist).query(q, k)
    ids, ds = orc.exact_topk(xo, qo, k, dist=dist)
    if dist == 3:
        assert np.max(np.abs(res["distance"] - ds)) <= 2 * (d + 3) * 2.0**-24 * np.max(ds)
        assert np.all(np.diff(res["distance"], axis=1) >= 0)
    else:
        assert np.array_equal(res["ID"], ids)
        assert np.array_equal(res["distance"], ds)


@pytest.mark.parametrize("n,nq,k,d,C", [
    (4000, 40, 32, 100, 4096),   # 128-byte quantised rows
    (2000, 33, 128, 120, 2048),  # the widest; the longest k
    (1000, 20, 1, 16, 1024),     # 32-byte rows
    (1000, 20, 10, 121, 1024),   # beyond them: every candidate is scored
    (3000, 20, 200, 50, 4096),   # k beyond them
])
@pytest.mark.parametrize("hard", [False, True])
def test_jaccard_bounds_rerank_equals_exact_scan(engine, n, nq, k, d, C, hard):
    """A list that holds the whole base re-ranks to the exact generalized-Jaccard scan, bit for
    bit: through the bounds, and where they leave too many candidates (copies of one row) or
    do not apply (a query with negative values)."""
    x, q = datasets.sparse_gamma(n, d, 101), datasets.sparse_gamma(nq, d, 102)
    if hard:
        x[::2] = x[0]
        q[::5] = x[0]
        q[3, : d // 2] = -2.5
        q[4] = 0
        q[4, 0] = 1e-6
    idx = engine.Index(x, implementation=10, distanceFunc=2, sketchDim=64, options=engine.make_options(candidates=C))
    ex = engine.Index(x, implementation=2, distanceFunc=2)
    assert idx.query(q, k).tobytes() == ex.query(q, k).tobytes()


@pytest.mark.parametrize("n,nq,k,d,hashes,tables", [
    (30000, 40, 32, 100, 2, 24),   # lists through the bounds
    (30000, 40, 128, 128, 2, 32),  # the longest k and widest rows
    (30000, 40, 10, 16, 2, 24),    # many candidates within the bounds: scored in full
    (30000, 30, 32, 37, 2, 24),    # rows without 16-byte loads: the fused kernel
])
@pytest.mark.parametrize("hard", [False, True])
def test_lsh_bounds_scoring_equals_oracle(engine, orc, n, nq, k, d, hashes, tables, hard):
    """LSH queries whose candidates are reduced by bounds return the oracle's walk and scoring of
    the same tables, bit for bit; copies of one row, which the bounds cannot separate, too."""
    x, q = data(n, nq, d, count=60)
    if hard:
        x[::3] = x[0]
        q[:10] = x[0]
    P = 1 << (d - 1).bit_length()
    bits = hashes * P.bit_length()
    idx = engine.Index(x, implementation=2, distanceFunc=1, framework=1, keysImplementation=7, bucketKeyBits=bits,
                       tables=tables, options=engine.make_options(cp_hashes=hashes))
    xn, qn = orc.normalize(x), orc.normalize(q)
    diag = engine.random_plus_minus(P * tables * 3 * hashes)
    okeys, oqk = (orc.crosspoly(v, P, tables, hashes, 3, diag) for v in (xn, qn))
    ooff, obk = orc.lsh_build(okeys, tables, 1 << bits)
    ids, ds = orc.lsh_query(xn, qn, oqk, tables, 1 << bits, ooff, obk, 0, 0, None, None, 0,
                            max(32, 1 << (k - 1).bit_length()), 1, k)
    res = idx.query(q, k)
    assert np.array_equal(res["ID"], ids)
    assert np.array_equal(res["distance"], ds)


@pytest.mark.parametrize("n,nq,k,d", [
    (4096, 4, 32, 100),     # the smallest base and batch that are filtered, the longest k of it
    (4097, 65, 1, 16),      # one point in the last tile, one query in the second block; the narrowest rows
    (8193, 9, 64, 101),     # the longest k of 512 candidates, of as many tiles as k; a padded word
    (30000, 33, 128, 99),   # the longest k
    (20001, 129, 10, 128),  # the widest rows
    (60000, 200, 16, 3),    # d below the filter: the FP32 scan
    (5000, 40, 40, 100),    # k beyond it at this size
    (5000, 40, 10, 129),    # d beyond it
])
@pytest.mark.parametrize("case", ["plain", "copies", "dense", "offset", "queries", "base"])
def test_jaccard_filter_equals_fp32_scan(engine, n, nq, k, d, case):
    """Ids and distances of the filtered exact Jaccard scan are the FP32 scan's bit for bit, also
    where the bounds leave too many candidates or none apply."""
    x, q = datasets.sparse_gamma(n, d, 111), datasets.sparse_gamma(nq, d, 112)
    if case == "copies":
        x[::2] = x[0]
        q[::3] = x[0]
    elif case == "dense":  # every distance near every other
        rng = np.random.default_rng(7)
        x, q = rng.random((n, d), dtype=np.float32), rng.random((nq, d), dtype=np.float32)
    elif case == "offset":  # a narrow range far from zero, queries beyond it on both sides
        rng = np.random.default_rng(8)
        x = 7 + 1e-3 * rng.random((n, d), dtype=np.float32)
        q = 7 + 2e-3 * rng.random((nq, d), dtype=np.float32) - np.float32(5e-4)
    elif case == "queries":
        q[0] = 0
        q[1, 0] = -0.5
        q[2, d - 1] = np.nan
        q[3] *= np.float32(1e6)
    elif case == "base":
        x[n - 1, 0] = -1.0
    idx = engine.Index(x, implementation=2, distanceFunc=2)
    want = idx.query(q, 129)[:, :k]  # k beyond the filter: the FP32 scan
    assert idx.query(q, k).tobytes() == want.tobytes()


def test_jaccard_filter_saved_index(engine, tmp_path):
    x, q = datasets.sparse_gamma(9000, D, 113), datasets.sparse_gamma(70, D, 114)
    idx = engine.Index(x, implementation=2, distanceFunc=2)
    path = str(tmp_path / "jaccard.lshg")
    idx.save(path)
    assert engine.Index.load(path).query(q, 32).tobytes() == idx.query(q, 32).tobytes()


@pytest.mark.parametrize("kw", [
    dict(implementation=8), dict(implementation=9), dict(implementation=2, distanceFunc=1),
    dict(implementation=2, distanceFunc=2), dict(implementation=3, sketchDim=8), dict(implementation=4, distanceFunc=2,
                                                                                     sketchDim=64),
], ids=["tc", "e4m3", "angular", "jaccard", "simhash", "minhash"])
def test_batches_enqueued_back_to_back(engine, kw):
    """Batches of several sizes down one stream without a wait, their queries written on that stream
    just before: kernels that may start early read nothing of the batch before."""
    import torch

    n, k = 20000, 10
    jac = kw.get("distanceFunc") == 2
    x, q = (datasets.sparse_gamma(n, D, 121), datasets.sparse_gamma(400, D, 122)) if jac else data(n, 400)
    idx = engine.Index(x, options=engine.make_options(candidates=128), **kw)
    sizes = [1, 130, 3, 400, 64, 257]
    want = [idx.query(np.roll(q, i, axis=0)[:m], k) for i, m in enumerate(sizes)]
    st = torch.cuda.Stream()
    host = torch.from_numpy(q).cuda()
    torch.cuda.synchronize()
    for _ in range(5):
        buf, outs = torch.empty_like(host), []
        with torch.cuda.stream(st):
            for i, m in enumerate(sizes):
                buf.copy_(torch.roll(host, i, 0))
                outs.append(torch.full((m, k, 2), -7, dtype=torch.int32, device="cuda"))
                idx.query_device_async(buf.data_ptr(), m, k, outs[-1].data_ptr(), st.cuda_stream)
        st.synchronize()
        idx.sync(st.cuda_stream)
        for o, w in zip(outs, want):
            assert o.cpu().numpy().tobytes() == w.tobytes()


@pytest.mark.parametrize("n,nq,words,C,impl", [
    (12000, 1, 1, 32, 3),      # one word of a chunk; one query
    (30001, 33, 5, 128, 3),    # rows of 8 words, 5 used; the last tile partly filled
    (120000, 64, 8, 256, 5),   # the largest batch read as packed words; a sampled prepass
    (120000, 65, 8, 256, 5),   # beyond it: E2M1 rows
    (150000, 7, 20, 1024, 3),  # three chunks, the last one half used; 8-point maxima
    (40000, 64, 32, 4096, 3),  # four chunks
])
def test_sketch_scan_packed_words_equal_popcount(engine, n, nq, words, C, impl):
    """Base tiles expanded from the packed sketches, and ties enough to overflow some queries, give
    the popcount scan's results."""
    x, q = (data(n, nq) if impl == 3 else (datasets.sparse_gamma(n, D, 131), datasets.sparse_gamma(nq, D, 132)))
    x[: n // 3] = x[0]
    q[0] = x[0]
    kw = dict(implementation=impl, sketchDim=words, **({} if impl == 3 else {"distanceFunc": 2}))
    res = [engine.Index(x, options=engine.make_options(candidates=C, sketch_scan=mode), **kw).query(q, 32)
           for mode in (TENSOR, POPCOUNT)]
    assert np.array_equal(res[0], res[1])


@pytest.mark.parametrize("impl,words,C", [(3, 2, 128), (3, 4, 1024), (5, 4, 2048), (4, 64, 128), (10, 64, 512)])
def test_listed_rescans_split_over_the_base(engine, impl, words, C):
    """Queries that tie with half of the base are rescanned in splits of it and merged."""
    n, nq = 50000, 5
    x, q = data(n, nq) if impl == 3 else (datasets.sparse_gamma(n, D, 141), datasets.sparse_gamma(nq, D, 142))
    x[: n // 2] = x[0]
    q[1] = q[3] = x[0]
    kw = dict(implementation=impl, sketchDim=words, **({} if impl == 3 else {"distanceFunc": 2}))
    res = [engine.Index(x, options=engine.make_options(candidates=C, sketch_scan=mode), **kw).query(q, 32)
           for mode in (TENSOR, POPCOUNT)]
    assert np.array_equal(res[0], res[1])


@pytest.mark.parametrize("nq", [3, 1500])
@pytest.mark.parametrize("C", [32, 64, 128])
def test_sketch_scan_short_lists_by_block_and_by_warp(engine, nq, C):
    x, q = data(20000, nq)
    res = [engine.Index(x, implementation=3, sketchDim=4,
                        options=engine.make_options(candidates=C, sketch_scan=mode)).query(q, 32)
           for mode in (TENSOR, POPCOUNT)]
    assert np.array_equal(res[0], res[1])


@pytest.mark.parametrize("nq", [1, 1024, 1025])  # the largest batch of SIMT signs at 32 words, the smallest beyond
def test_simhash_signs_by_batch_size_equal_oracle(engine, orc, nq):
    x, q = data(3000, nq)
    idx = engine.Index(x, implementation=3, sketchDim=32)
    sk, _ = idx.sketch_queries(q, np.uint32, 32)
    assert np.array_equal(sk, orc.simhash(q, engine.random_normals(D * 32 * 32), 32, 32))
