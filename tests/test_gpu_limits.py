"""Queries at the limits of a device's memory and of several host threads: what a batch allocates,
what it does where its optional temporaries do not fit, and indexes of different dimensions
queried at the same time.

Memory is limited by a pool with a maximum size of its own, in place of the device's default
pool, so the device itself is never filled.
"""
import contextlib
import ctypes as C
import threading

import numpy as np
import pytest

from lshongpu_gb300 import datasets

pytestmark = pytest.mark.gpu

USED_HIGH = 0x8  # cudaMemPoolAttrUsedMemHigh


class PoolProps(C.Structure):
    """struct cudaMemPoolProps."""
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location_type", C.c_int),
                ("location_id", C.c_int), ("security", C.c_void_p), ("max_size", C.c_size_t),
                ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


def cudart():
    import torch

    torch.cuda.synchronize()
    rt = C.CDLL("libcudart.so.13")
    rt.cudaMemPoolDestroy.argtypes = [C.c_void_p]
    rt.cudaDeviceSetMemPool.argtypes = [C.c_int, C.c_void_p]
    for f in ("cudaMemPoolGetAttribute", "cudaMemPoolSetAttribute"):
        getattr(rt, f).argtypes = [C.c_void_p, C.c_int, C.c_void_p]
    return rt


@contextlib.contextmanager
def memory_pool(max_bytes=0):
    """The device's allocations come from a pool of at most max_bytes (0: no limit of its own);
    yields a function that returns, and resets, the most bytes in use since its last call."""
    rt = cudart()
    old, pool = C.c_void_p(), C.c_void_p()
    assert rt.cudaDeviceGetMemPool(C.byref(old), 0) == 0
    props = PoolProps(alloc_type=1, location_type=1, location_id=0, max_size=max_bytes)
    assert rt.cudaMemPoolCreate(C.byref(pool), C.byref(props)) == 0
    assert rt.cudaDeviceSetMemPool(0, pool) == 0

    def high():
        v = C.c_uint64()
        assert rt.cudaDeviceSynchronize() == 0
        assert rt.cudaMemPoolGetAttribute(pool, USED_HIGH, C.byref(v)) == 0
        zero = C.c_uint64(0)
        assert rt.cudaMemPoolSetAttribute(pool, USED_HIGH, C.byref(zero)) == 0
        return v.value

    try:
        yield high
    finally:
        rt.cudaDeviceSynchronize()
        assert rt.cudaDeviceSetMemPool(0, old) == 0
        assert rt.cudaMemPoolDestroy(pool) == 0


def test_lsh_batch_without_room_for_the_bounds(engine):
    """An LSH batch whose candidate lists fit, but not the 2 KB a query its bounds keep, is scored
    without them, with the same results."""
    n, d, nq = 20000, 16, 43000
    x = datasets.clustered(n, d, 151, count=200)
    q = np.tile(datasets.clustered(1000, d, 152, count=200), (nq // 1000, 1))
    kw = dict(implementation=2, distanceFunc=1, framework=1, keysImplementation=7, bucketKeyBits=10, tables=7,
              options=engine.make_options(cp_hashes=2))
    with memory_pool() as high:
        idx = engine.Index(x, **kw)
        high()
        want = idx.query(q, 32)
        full = high()
        idx.close()
    kept = nq * 2048
    with memory_pool(full - kept // 2) as high:
        idx = engine.Index(x, **kw)
        got = idx.query(q, 32)
        idx.close()
    assert got.tobytes() == want.tobytes()


@pytest.mark.parametrize("dist,k", [(1, 32), (2, 10), (1, 200)])
def test_two_threads_of_different_dimensions(engine, dist, k):
    """Host threads that query indexes of 20 and of 128 dimensions at the same time: the kernels they
    share are launched with different amounts of shared memory."""
    import torch

    batches, nq = 3000, 8
    jobs = []
    for d in (20, 128):
        rows = datasets.sparse_gamma if dist == 2 else datasets.clustered
        x, q = rows(4200, d, 161), rows(nq, d, 162)
        idx = engine.Index(x, implementation=2, distanceFunc=dist)
        jobs.append((idx, idx.query(q, k), torch.from_numpy(q).cuda(), torch.cuda.Stream(),
                     torch.empty((nq, k, 2), dtype=torch.int32, device="cuda")))
    torch.cuda.synchronize()
    failed = []
    start = threading.Barrier(len(jobs))

    def work(idx, want, q, stream, out):
        start.wait()
        try:
            for _ in range(batches):
                idx.query_device_async(q.data_ptr(), nq, k, out.data_ptr(), stream=stream.cuda_stream)
            idx.sync(stream.cuda_stream)
            if out.cpu().numpy().tobytes() != want.tobytes():
                failed.append("results differ")
        except engine.LshgError as e:
            failed.append(str(e))

    threads = [threading.Thread(target=work, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.mark.parametrize("n,dist", [(60000, 1), (60000, 2), (1000000, 2)])
def test_exact_batches_allocate_by_the_query(engine, n, dist):
    """A filtered exact batch takes less than 32 KB a query and 16 MB, also on a large base: the rescan of
    listed queries has no lists of its own, whose number was as large as if every query were listed
    alone, and the Jaccard scan's group maxima are bounded."""
    d, nq = 16, 1000
    rows = datasets.sparse_gamma if dist == 2 else datasets.clustered
    x, q = rows(n, d, 171), rows(nq, d, 172)
    with memory_pool() as high:
        idx = engine.Index(x, implementation=2, distanceFunc=dist)
        high()
        held = high()
        idx.query(q, 100)
        used = high() - held
        idx.close()
    assert used <= nq * 32768 + (16 << 20)


@pytest.mark.parametrize("dist", [1, 2])
@pytest.mark.parametrize("n,nq,listed,d,k", [
    (4096, 4, 1, 16, 1),          # one listed query, one neighbour; few tiles a split
    (9000, 200, 3, 37, 64),       # listed queries anywhere in the batch; lists of 64
    (20011, 70, 65, 100, 32),     # a second block of one query
    (30000, 1500, 1500, 20, 10),  # every query: few splits
    (50000, 300, 299, 128, 128),  # lists of 128, one CTA an SM
])
def test_listed_queries_equal_fp32_scan(engine, dist, n, nq, listed, d, k):
    """Queries that tie with a third of the base, or (angular) have no direction, are scanned in full within
    the limits their scores give: ids and distances of the FP32 scan, bit for bit."""
    rows = datasets.sparse_gamma if dist == 2 else datasets.clustered
    x, q = rows(n, d, 181), rows(nq, d, 182)
    x[1::3] = x[0]
    at = np.random.default_rng(5).permutation(nq)[:listed]
    q[at] = x[0]
    q[at[1::3]] *= np.float32(1.0003)
    q[at[2::7]] = 0 if dist == 1 else q[at[2::7]]
    idx = engine.Index(x, implementation=2, distanceFunc=dist)
    want = idx.query(q, 129)[:, :k]  # k beyond the filter: the FP32 scan
    assert idx.query(q, k).tobytes() == want.tobytes()


@pytest.mark.parametrize("n,d,filtered", [
    (5000, 1, False), (5000, 2, False), (32768, 3, True), (32769, 3, False), (131072, 4, True), (131073, 4, False),
    (200000, 5, True), (200000, 6, True),
])
def test_exact_filter_at_few_dimensions(engine, n, d, filtered):
    """On a sphere of few dimensions the scores' error holds more points than the filter has places from
    some base size on: the FP32 scan answers those, with the same results."""
    rng = np.random.default_rng(7)
    x, q = (rng.standard_normal((m, d)).astype(np.float32) for m in (n, 70))
    idx = engine.Index(x, implementation=2, distanceFunc=1)
    engine.profile_enable(True)
    engine.profile_report()
    got = idx.query(q, 32)
    ran = engine.profile_report()
    engine.profile_enable(False)
    assert ("tc_filter" in ran) == filtered
    assert got.tobytes() == idx.query(q, 129)[:, :32].tobytes()  # k beyond the filter: the FP32 scan


@pytest.mark.parametrize("case,filtered", [("sparse", True), ("dense", True), ("copies of 1000", True),
                                           ("a third copies", True), ("copies of 10", False), ("near rows", False)])
def test_jaccard_filter_by_the_bases_resolution(engine, case, filtered):
    """A base whose rows have, mostly, more points within the codes' resolution than a query has places
    is left to the FP32 scan; results are its either way."""
    n, d, nq, k = 60013, 100, 40, 10
    rng = np.random.default_rng(9)
    x, q = datasets.sparse_gamma(n, d, 191), datasets.sparse_gamma(nq, d, 192)
    if case == "dense":
        x, q = rng.random((n, d), dtype=np.float32), rng.random((nq, d), dtype=np.float32)
    elif case == "a third copies":
        x[::3] = x[0]
    elif case.startswith("copies of"):
        x = x[rng.integers(0, int(case.split()[-1]), n)]
    elif case == "near rows":
        x, q = (x[:1] + 1e-4 * rng.random((m, d), dtype=np.float32) for m in (n, nq))
    idx = engine.Index(x, implementation=2, distanceFunc=2)
    engine.profile_enable(True)
    engine.profile_report()
    got = idx.query(q, k)
    ran = engine.profile_report()
    engine.profile_enable(False)
    assert ("jaccard_filter" in ran) == filtered
    assert got.tobytes() == idx.query(q, 129)[:, :k].tobytes()  # k beyond the filter: the FP32 scan


@pytest.mark.parametrize("n,nq,k", [
    (196608, 9, 100),  # 6,144 group maxima: a tile a group
    (196609, 70, 32),  # one point more: two tiles a group, the last group of one tile
    (450000, 33, 128),  # three
    (700000, 5, 10),   # a sampled pass of them
])
def test_jaccard_filter_groups_of_tiles(engine, n, nq, k):
    """Bases with more group maxima than the threshold select takes: the FP32 scan's results."""
    x, q = datasets.sparse_gamma(n, 20, 201), datasets.sparse_gamma(nq, 20, 202)
    idx = engine.Index(x, implementation=2, distanceFunc=2)
    assert idx.query(q, k).tobytes() == idx.query(q, 129)[:, :k].tobytes()  # k beyond the filter


@pytest.mark.parametrize("impl,n,nq,d,C,k", [
    (3, 20000, 40, 64, 1024, 10),     # rows staged in shared memory
    (3, 20000, 33, 128, 4096, 128),   # the widest rows, the longest list and k
    (3, 20000, 700, 37, 2048, 32),    # rows read directly; several queries a block
    (6, 20000, 20, 100, 1024, 1),
    (10, 20000, 400, 40, 4096, 32),   # Jaccard
    (10, 20000, 17, 33, 1024, 100),   # Jaccard, read directly
])
def test_listed_rerank_equals_full_rerank(engine, impl, n, nq, d, C, k):
    """Lists that the 8-bit bounds cannot separate (near-equal rows), all of a batch and some of one: what
    scoring every candidate returns."""
    rng = np.random.default_rng(11)
    rows = datasets.sparse_gamma if impl == 10 else datasets.clustered
    x, q = rows(n, d, 211), rows(nq, d, 212)
    near = lambda m: np.abs(x[:1] + 1e-4 * rng.standard_normal((m, d))).astype(np.float32) if impl == 10 else \
        (x[:1] + 1e-4 * rng.standard_normal((m, d))).astype(np.float32)
    x[: n // 2] = near(n // 2)
    kw = dict(implementation=impl, sketchDim=64 if impl == 10 else 8, options=engine.make_options(candidates=C))
    idx = engine.Index(x, **kw, **({"distanceFunc": 2} if impl == 10 else {}))
    for some in (q, near(nq)):
        some[::3] = near(len(some[::3]))
        want = idx.query(some, 129)[:, :k]  # k beyond the bounds: every candidate is scored
        assert idx.query(some, k).tobytes() == want.tobytes()


@pytest.mark.parametrize("sigma,copies,used", [(0.05, 1, True), (0.05, 50, True), (0.01, 1, False), (0.05, 2000, False)])
def test_lsh_bounds_by_the_bases_resolution(engine, sigma, copies, used):
    """LSH candidates go through bounds unless the base's rows mostly have more points within the codes'
    resolution than a query may keep; results are those of scoring every candidate either way."""
    n, d, nq, k = 100000, 100, 200, 32
    x = datasets.clustered(n // copies, d, 221, count=50, sigma=sigma)
    q = datasets.clustered(nq, d, 222, count=50, sigma=sigma)
    x = np.ascontiguousarray(np.repeat(x, copies, axis=0))
    idx = engine.Index(x, implementation=2, distanceFunc=1, framework=1, keysImplementation=7, bucketKeyBits=16,
                       tables=80, options=engine.make_options(cp_hashes=2))
    engine.profile_enable(True)
    engine.profile_report()
    got = idx.query(q, k)
    ran = engine.profile_report()
    engine.profile_enable(False)
    assert ("rerank_bounds" in ran) == used
    assert got.tobytes() == idx.query(q, 129)[:, :k].tobytes()  # k beyond the bounds


@pytest.mark.parametrize("n,nq,k,d,tables,used", [
    (80000, 200, 32, 100, 98, False),  # 119 entries a query on average
    (80000, 200, 32, 100, 99, True),   # 120
    (8000, 3, 128, 16, 16, False),     # 125, 375 in the batch
    (8000, 4, 128, 16, 16, True),      # 500
    (4000, 1, 1, 128, 256, False),     # 15
    (27000, 1, 10, 16, 16, True),      # 421, one query
    (200000, 50, 10, 16, 16, False),   # 3,125: more than half of the list's places
])
def test_lsh_bounds_rule(engine, n, nq, k, d, tables, used):
    """Where LSH candidates go through bounds, and that the results do not depend on it."""
    x, q = datasets.clustered(n, d, 231, count=500), datasets.clustered(nq, d, 232, count=500)
    P = 1 << (d - 1).bit_length()
    idx = engine.Index(x, implementation=2, distanceFunc=1, framework=1, keysImplementation=7,
                       bucketKeyBits=2 * P.bit_length(), tables=tables, options=engine.make_options(cp_hashes=2))
    engine.profile_enable(True)
    engine.profile_report()
    got = idx.query(q, k)
    ran = engine.profile_report()
    engine.profile_enable(False)
    assert ("rerank_bounds" in ran) == used
    assert got.tobytes() == idx.query(q, 129)[:, :k].tobytes()  # k beyond the bounds
