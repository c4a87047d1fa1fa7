"""Product-quantised batches on the tensor-core path (code rows decoded to fp16 operand rows, contracted, listed rows
re-scored from the distance tables): ids and distances equal the CPU oracle's table sums bit for bit."""
import numpy as np
import pytest

from parity import logged_launches

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vsk():
    import vectorstorekit_b200 as v
    return v


@pytest.fixture(scope="module")
def dev(vsk):
    return vsk.CUDAAcceleratorStrategy(0).initialize()


def _index(vsk, dev, cb, codes):
    m, ksub, ds = cb.shape
    pq = vsk.ProductQuantizer(dev, m * ds, segments=m, codeSize=int(np.log2(ksub)))
    pq.set_codebooks(cb)
    ix = pq.index()
    ix.add(codes)
    return ix


def _clustered(rng, n, nq, m, ksub, ds, offset=0.0, noise=0.3):
    """Rows and queries around 64 centres; codewords are segments of sampled rows."""
    d = m * ds
    centres = rng.standard_normal((64, d)).astype(np.float32) + np.float32(offset)
    x = (centres[rng.integers(0, 64, n)] + noise * rng.standard_normal((n, d))).astype(np.float32)
    q = (centres[rng.integers(0, 64, nq)] + noise * rng.standard_normal((nq, d))).astype(np.float32)
    cb = np.stack([x[rng.choice(n, ksub, replace=False)][:, s * ds:(s + 1) * ds] for s in range(m)])
    return q, np.ascontiguousarray(cb), x


# (n, m, ds, ksub, nq, k): the smallest batch and index of the path, partial query and row tiles, every segment length
# with a decode path of its own (2, 4, multiples of 8) and others, operand widths with the row term folded in (inside
# the padding, d = 40; in a block of its own, d = 64 and 256) and in the epilogue (d = 320), k to the path's limit
@pytest.mark.parametrize("shape", [(16_384, 8, 8, 256, 64, 10), (16_385, 16, 8, 256, 129, 1), (40_001, 8, 2, 256, 65, 37),
                                   (30_000, 16, 4, 256, 300, 100), (20_001, 5, 8, 16, 128, 10), (20_000, 16, 16, 256, 70, 10),
                                   (20_000, 10, 32, 64, 70, 10), (17_000, 7, 3, 256, 200, 5), (17_001, 24, 1, 16, 90, 10),
                                   (50_000, 8, 8, 256, 64, 1024), (17_777, 32, 24, 16, 100, 10)])
def test_tensor_batches_equal_table_sums(vsk, dev, cpu_oracle, shape):
    n, m, ds, ksub, nq, k = shape
    rng = np.random.default_rng(n + m + nq)
    q, cb, x = _clustered(rng, n, nq, m, ksub, ds)
    codes = cpu_oracle.pq_encode(x, cb)
    ix = _index(vsk, dev, cb, codes)
    before = dev.stats()["tensor_tiles"]
    dist, ids = ix.batchSearch(q, k)
    assert dev.stats()["tensor_tiles"] > before
    rd, ri = cpu_oracle.pq_search(q, codes, cb, k)
    assert np.array_equal(ids, ri)
    assert np.array_equal(dist, rd)
    # one query fewer than the path takes: the table scan gives the same rows
    d1, i1 = ix.batchSearch(q[:63], k)
    assert np.array_equal(i1, ri[:63]) and np.array_equal(d1, rd[:63])


# tables of sixteen queries to a block (from 256 queries on): every segment length with a kernel of its own, one of the general
# kernel, remainders of 0, 1 and 15 queries, few codewords; and operand rows of 128, 129 and more 16-byte pieces
@pytest.mark.parametrize("m,ds,ksub,nq", [(8, 2, 256, 256), (8, 4, 256, 257), (8, 8, 32, 271), (4, 16, 256, 255), (4, 16, 256, 256),
                                          (8, 3, 256, 272), (63, 16, 16, 64), (129, 8, 16, 64), (131, 8, 16, 70)])
def test_tables_and_wide_rows(vsk, dev, cpu_oracle, m, ds, ksub, nq):
    rng = np.random.default_rng(m * ds + nq)
    q, cb, x = _clustered(rng, 16_411, nq, m, ksub, ds)
    codes = cpu_oracle.pq_encode(x, cb)
    ix = _index(vsk, dev, cb, codes)
    before = dev.stats()["tensor_tiles"]
    dist, ids = ix.batchSearch(q, 10)
    assert dev.stats()["tensor_tiles"] > before
    rd, ri = cpu_oracle.pq_search(q, codes, cb, 10)
    assert np.array_equal(ids, ri)
    assert np.array_equal(dist, rd)


@pytest.mark.parametrize("offset", [30.0, 3000.0])
def test_rows_far_from_the_origin(vsk, dev, cpu_oracle, offset):
    """The error bound grows with the rows' norms: lists get longer, and where they overflow the table scan answers."""
    rng = np.random.default_rng(5)
    q, cb, x = _clustered(rng, 30_000, 80, 8, 256, 4, offset)
    codes = cpu_oracle.pq_encode(x, cb)
    ix = _index(vsk, dev, cb, codes)
    dist, ids = ix.batchSearch(q, 20)
    rd, ri = cpu_oracle.pq_search(q, codes, cb, 20)
    assert np.array_equal(ids, ri) and np.array_equal(dist, rd)


def test_bulk_ties_and_late_block_fall_back(vsk, dev, cpu_oracle):
    rng = np.random.default_rng(6)
    n, m, ds = 60_000, 2, 4
    cb = rng.standard_normal((m, 16, ds)).astype(np.float32)
    q = rng.standard_normal((70, m * ds)).astype(np.float32)
    codes = rng.integers(0, 4, (n, m)).astype(np.uint8)          # 16 distinct rows: thousands tie at every distance
    dist, ids = _index(vsk, dev, cb, codes).batchSearch(q, 100)
    rd, ri = cpu_oracle.pq_search(q, codes, cb, 100)
    assert np.array_equal(ids, ri) and np.array_equal(dist, rd)
    codes = rng.integers(0, 6, (n, m)).astype(np.uint8)
    codes[n - 20_000:] = (7, 11)                                  # the nearest row of half the queries, late and in bulk
    q[::2] = np.concatenate([cb[0, 7], cb[1, 11]]) + 0.01 * rng.standard_normal((35, m * ds)).astype(np.float32)
    dist, ids = _index(vsk, dev, cb, codes).batchSearch(q, 100)
    rd, ri = cpu_oracle.pq_search(q, codes, cb, 100)
    assert np.array_equal(ids, ri) and np.array_equal(dist, rd)


def test_non_finite_queries_do_not_disturb_the_others(vsk, dev, cpu_oracle):
    rng = np.random.default_rng(7)
    q, cb, x = _clustered(rng, 20_000, 80, 8, 256, 4)
    codes = cpu_oracle.pq_encode(x, cb)
    ix = _index(vsk, dev, cb, codes)
    rd, ri = cpu_oracle.pq_search(q, codes, cb, 10)
    bad = q.copy()
    bad[3, 5], bad[70, 0] = np.nan, np.inf
    dist, ids = ix.batchSearch(bad, 10)
    keep = [i for i in range(80) if i not in (3, 70)]
    assert np.array_equal(ids[keep], ri[keep]) and np.array_equal(dist[keep], rd[keep])
    # a codebook with an infinite entry has no fp16 form: the table scan takes the batch
    cb2 = cb.copy()
    cb2[0, 9, 0] = np.inf
    before = dev.stats()["tensor_tiles"]
    dist, ids = _index(vsk, dev, cb2, codes).batchSearch(q, 10)
    assert dev.stats()["tensor_tiles"] == before
    rd, ri = cpu_oracle.pq_search(q, codes, cb2, 10)
    assert np.array_equal(ids, ri) and np.array_equal(dist, rd)


def test_ordinary_batches_are_answered_by_the_contraction(vsk, dev, cpu_oracle):
    """Not by the table scan behind it: no query is handed back."""
    for m, ds in ((16, 8), (10, 32)):                             # queries resident, and the general kernel
        rng = np.random.default_rng(m)
        q, cb, x = _clustered(rng, 30_000, 100, m, 256, ds)
        codes = cpu_oracle.pq_encode(x, cb)
        ix = _index(vsk, dev, cb, codes)
        before = dev.stats()["fallback_queries"]
        (dist, ids), names = logged_launches(dev, lambda: ix.batchSearch(q, 10))
        assert ("list_scan" if m == 16 else "scan") in names
        assert dev.stats()["fallback_queries"] == before
        rd, ri = cpu_oracle.pq_search(q, codes, cb, 10)
        assert np.array_equal(ids, ri) and np.array_equal(dist, rd)


def test_an_index_of_bulk_ties_rests_from_the_contraction(vsk, dev, cpu_oracle):
    rng = np.random.default_rng(16)
    n, m, ds = 60_000, 2, 4
    cb = rng.standard_normal((m, 16, ds)).astype(np.float32)
    q = rng.standard_normal((150, m * ds)).astype(np.float32)
    codes = rng.integers(0, 3, (n, m)).astype(np.uint8)          # 9 distinct rows
    ix = _index(vsk, dev, cb, codes)
    rd, ri = cpu_oracle.pq_search(q, codes, cb, 100)
    decoded = []
    for _ in range(17):
        (dist, ids), names = logged_launches(dev, lambda: ix.batchSearch(q, 100))
        decoded.append("pq_decode" in names)
        assert np.array_equal(ids, ri) and np.array_equal(dist, rd)
    assert decoded == [True] + [False] * 15 + [True]


def test_entries_of_nearly_equal_size(vsk, dev, cpu_oracle):
    """Vectors in the positive quadrant: the thresholds lie near half the largest squared norm, the far end of what the operand
    columns hold.  The contraction still answers."""
    rng = np.random.default_rng(17)
    m, ds, n, nq = 16, 8, 30_000, 100
    x = rng.uniform(0.5, 1.0, (n, m * ds)).astype(np.float32)
    q = rng.uniform(0.5, 1.0, (nq, m * ds)).astype(np.float32)
    cb = np.ascontiguousarray(np.stack([x[rng.choice(n, 256, replace=False)][:, s * ds:(s + 1) * ds] for s in range(m)]))
    codes = cpu_oracle.pq_encode(x, cb)
    ix = _index(vsk, dev, cb, codes)
    before = dev.stats()["fallback_queries"]
    dist, ids = ix.batchSearch(q, 10)
    rd, ri = cpu_oracle.pq_search(q, codes, cb, 10)
    assert np.array_equal(ids, ri) and np.array_equal(dist, rd)
    assert dev.stats()["fallback_queries"] == before


# segment lengths with the short form; codebooks of a size that fills no warp; rows far from the origin, rows far from every
# codeword, rows at equal distances from two codewords, and rows that are not finite
@pytest.mark.parametrize("ds,ksub", [(4, 256), (8, 256), (16, 256), (8, 33), (16, 2)])
@pytest.mark.parametrize("offset", [0.0, 10.0, 1e4])
def test_encoding_equals_the_exact_sums(vsk, dev, cpu_oracle, ds, ksub, offset):
    rng = np.random.default_rng(ds + ksub)
    m, n = 3, 5_003
    x = (rng.standard_normal((n, m * ds)) + offset * rng.standard_normal(m * ds)).astype(np.float32)
    cb = np.ascontiguousarray(np.stack([x[rng.choice(n, ksub, replace=False)][:, s * ds:(s + 1) * ds] for s in range(m)]))
    cb[:, ksub - 1] = cb[:, 0]                                    # equal codewords: the lower code
    x[11] *= 1e3
    x[12] *= 1e18                                                 # squares that overflow
    x[13, 1], x[14, 2] = np.nan, np.inf
    x[15] = 0.5 * (np.concatenate(list(cb[:, 0])) + np.concatenate(list(cb[:, 1])))
    assert np.array_equal(_encode(dev, cb, x), cpu_oracle.pq_encode(x, cb))


# The contraction takes 129 or more codewords from 65 536 (row, segment) pairs on (131 072 for two dimensions): whole and ragged
# row tiles, whole and partial groups of segments.
@pytest.mark.parametrize("ds,m,ksub,n", [(2, 8, 256, 16_384), (2, 10, 129, 13_185), (4, 8, 256, 8_319), (4, 9, 200, 8_000), (8, 4, 256, 20_001),
                                         (8, 5, 255, 13_185), (8, 16, 256, 19_072), (16, 2, 256, 32_896), (16, 3, 130, 22_007),
                                         # rows narrower than the 32 (16) columns that are fetched of them
                                         (2, 2, 256, 65_537), (4, 2, 200, 33_001), (8, 2, 256, 32_896), (8, 3, 129, 22_003), (16, 1, 256, 65_600)])
def test_encoding_on_the_tensor_cores_equals_the_exact_sums(vsk, dev, cpu_oracle, ds, m, ksub, n):
    rng = np.random.default_rng(ds * 100 + m)
    x = (rng.standard_normal((n, m * ds)) + 2.0 * rng.standard_normal(m * ds)).astype(np.float32)
    cb = np.ascontiguousarray(np.stack([x[rng.choice(n, ksub, replace=False)][:, s * ds:(s + 1) * ds] for s in range(m)]))
    cb[:, ksub - 1] = cb[:, 3]                                    # equal codewords: the lower code
    cb[m - 1, 7] *= 40.0                                          # one far out: the others share few operand bits
    x[5] = np.concatenate(list(cb[:, 3]))
    x[6] = 0.5 * (np.concatenate(list(cb[:, 0])) + np.concatenate(list(cb[:, 1])))
    for i in range(100):                                          # between two codewords, in one four or in two
        a, b = (2 * i) % (ksub - 2), (2 * i + (1 if i % 2 else 17)) % (ksub - 2)
        x[20 + i] = 0.5 * (np.concatenate(list(cb[:, a])) + np.concatenate(list(cb[:, b])))
    x[7] *= 1e4                                                   # more than fp16 holds beside the codewords
    x[8] *= 1e19                                                  # squares that overflow
    x[9, 1], x[10, 0] = np.nan, np.inf
    x[n - 1] = x[5]
    assert np.array_equal(_encode(dev, cb, x), cpu_oracle.pq_encode(x, cb))


@pytest.mark.parametrize("what", ["equal", "tiny", "huge", "largest", "nan"])
def test_encoding_with_unusual_codebooks(vsk, dev, cpu_oracle, what):
    rng = np.random.default_rng(8)
    m, ksub, ds, n = 5, 256, 8, 13_200
    x = rng.standard_normal((n, m * ds)).astype(np.float32)
    cb = rng.standard_normal((m, ksub, ds)).astype(np.float32)
    if what == "equal":
        cb[1] = cb[1, 0]
    elif what == "tiny":
        cb[1] *= np.float32(1e-41)
        x[:, ds:2 * ds] *= np.float32(1e-41)
    elif what == "huge":
        cb[1] *= np.float32(1e20)
        x[:, ds:2 * ds] *= np.float32(1e18)
    elif what == "largest":                                       # one codeword of every four near fp32's limit, the mean is not
        cb[1] *= np.float32(1e37)
        big = np.arange(0, ksub, 4)
        cb[1, big] = np.where(big // 32 % 2, -1, 1)[:, None] * (2.9e38 * (1 + 0.01 * rng.random((len(big), ds)))).astype(np.float32)
        x[:, ds:2 * ds] = cb[1, rng.integers(0, ksub, n)]
    else:
        cb[1, 9, 3], cb[2, 200, 0] = np.nan, np.inf
    assert np.array_equal(_encode(dev, cb, x), cpu_oracle.pq_encode(x, cb))


def _encode(dev, cb, x):
    """vsk_pq_encode with a codebook size that need not be a power of two."""
    import ctypes as C
    m, ksub, ds = cb.shape
    codes = np.empty((x.shape[0], m), np.uint8)
    dev.check(dev._lib.vsk_pq_encode(dev._h, cb.ctypes.data_as(C.c_void_p), m * ds, m, ksub, x.ctypes.data_as(C.c_void_p),
                                     x.shape[0], codes.ctypes.data_as(C.c_void_p)))
    return codes


def test_a_bounded_wait_of_the_row_lists_runs_out(vsk, cpu_oracle):
    dev = vsk.CUDAAcceleratorStrategy(0).initialize()
    try:
        rng = np.random.default_rng(42)
        q, cb, x = _clustered(rng, 40_000, 100, 16, 256, 8)
        codes = cpu_oracle.pq_encode(x, cb)
        ix = _index(vsk, dev, cb, codes)
        dev.set_tuning(wait_limit_log2=16, test_stall_scan=1)
        with pytest.raises(vsk.Timeout):
            ix.batchSearch(q, 10)
        assert dev.tuning()["test_stall_scan"] == 0
        dev.set_tuning(wait_limit_log2=0)
        dist, ids = ix.batchSearch(q, 10)
        rd, ri = cpu_oracle.pq_search(q, codes, cb, 10)
        assert np.array_equal(ids, ri) and np.array_equal(dist, rd)
        ix.close()
    finally:
        dev.close()
