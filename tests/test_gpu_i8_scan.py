"""dotProduct batches over int8 codes on the integer contraction (8-bit queries, exact accumulators, listed rows re-scored
against the dequantised rows): the rows the CPU oracle finds, for operand widths around its K blocks and TMA strides."""
import numpy as np
import pytest

import oracle
from parity import assert_topk_parity, logged_launches

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vsk():
    import vectorstorekit_b200 as v
    return v


@pytest.fixture(scope="module")
def dev(vsk):
    return vsk.CUDAAcceleratorStrategy(0).initialize()


def _quantised(vsk, dev, x):
    """(index, codes, scale, offset) of the rows, quantised per dimension."""
    quantizer = vsk.ScalarQuantizer(dev, per_dim=True)
    quantizer.train(x)
    codes = quantizer.quantizeBatch(x)
    ix = vsk.QuantizedFlatIndex(dev, x.shape[1], vsk.DistanceMetric.dotProduct, quantizer.scale, quantizer.offset)
    ix.add(codes)
    return ix, np.asarray(codes), np.asarray(quantizer.scale, np.float32), np.asarray(quantizer.offset, np.float32)


def _check(cpu_oracle, ix, codes, scale, offset, q, k):
    d, i = ix.batchSearch(q, k)
    rd, ri = cpu_oracle.sq8_search(oracle.DOT, q, codes, scale, offset, k)
    assert_topk_parity(d, i, rd, ri)


# one and several K blocks of 128 codes, partial 32-byte steps, rows padded for TMA (dim not a multiple of 16), the
# smallest index of the path, partial tiles, one query, k up to the path's limit
@pytest.mark.parametrize("shape", [(16_384, 128, 128, 10), (16_385, 129, 1, 10), (20_000, 16, 300, 37), (20_001, 33, 65, 1),
                                   (30_000, 384, 200, 10), (17_003, 250, 130, 100), (16_400, 513, 9, 10), (40_000, 64, 64, 1024)])
def test_integer_contraction_finds_the_oracles_rows(vsk, dev, cpu_oracle, shape):
    n, d, nq, k = shape
    rng = np.random.default_rng(n + d + nq)
    x = rng.standard_normal((n, d)).astype(np.float32) * rng.uniform(0.2, 3.0, d).astype(np.float32) + rng.normal(0, 1, d).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    ix, codes, scale, offset = _quantised(vsk, dev, x)
    before = dev.stats()["tensor_tiles"]
    _check(cpu_oracle, ix, codes, scale, offset, q, k)
    assert dev.stats()["tensor_tiles"] > before
    # rows added later are seen
    ix.add(codes[:257])
    _check(cpu_oracle, ix, np.concatenate([codes, codes[:257]]), scale, offset, q, k)


def test_lists_that_overflow_go_to_the_other_paths(vsk, dev, cpu_oracle):
    """Rows of one direction and many norms, in ascending order of their products: every later row passes the bar.  The
    answer is the same, on the batch's first search and on the ones after it."""
    rng = np.random.default_rng(8)
    n, d = 30_000, 48
    base = rng.standard_normal(d).astype(np.float32)
    x = np.linspace(0.01, 1.0, n, dtype=np.float32)[:, None] * base + 1e-3 * rng.standard_normal((n, d)).astype(np.float32)
    ix, codes, scale, offset = _quantised(vsk, dev, x)
    q = (base + 0.1 * rng.standard_normal((300, d))).astype(np.float32)
    for _ in range(2):
        _check(cpu_oracle, ix, codes, scale, offset, q, 20)
    q[7, 3] = np.inf
    q[9] = 0.0
    d_, i_ = ix.batchSearch(q, 20)
    keep = [i for i in range(300) if i not in (7, 9)]
    rd, ri = cpu_oracle.sq8_search(oracle.DOT, q[keep], codes, scale, offset, 20)
    assert_topk_parity(d_[keep], i_[keep], rd, ri)


# resident query block (up to three K blocks) and the general kernel beyond it; the integer path answers by itself
@pytest.mark.parametrize("shape", [(20_000, 64, 100, 10), (20_000, 384, 300, 10), (17_000, 513, 70, 10), (16_385, 129, 1, 10)])
def test_the_integer_contraction_answers_ordinary_batches(vsk, dev, cpu_oracle, shape):
    n, d, nq, k = shape
    rng = np.random.default_rng(n + d)
    ix, codes, scale, offset = _quantised(vsk, dev, rng.standard_normal((n, d)).astype(np.float32))
    q = rng.standard_normal((nq, d)).astype(np.float32)
    before = dev.stats()["fallback_queries"]
    (got, names) = logged_launches(dev, lambda: ix.batchSearch(q, k))
    assert "query_operands" not in names                          # (the fp16 path's first launch)
    assert ("list_scan" in names) == (d <= 384) and ("scan" in names) == (d > 384)
    assert dev.stats()["fallback_queries"] == before
    assert_topk_parity(*got, *cpu_oracle.sq8_search(oracle.DOT, q, codes, scale, offset, k))


def test_a_few_degenerate_queries_decide_for_themselves_only(vsk, dev, cpu_oracle):
    """Zero vectors tie with every row and non-finite ones have no 8-bit form: they are re-run one by one, their batch keeps its
    results and the batches after it their path."""
    rng = np.random.default_rng(21)
    ix, codes, scale, offset = _quantised(vsk, dev, rng.standard_normal((20_000, 64)).astype(np.float32))
    q = rng.standard_normal((100, 64)).astype(np.float32)
    rd, ri = cpu_oracle.sq8_search(oracle.DOT, q, codes, scale, offset, 10)
    bad = q.copy()
    bad[3], bad[50] = 0.0, 0.0
    bad[60, 1], bad[61, 2] = np.nan, np.inf
    keep = [i for i in range(100) if i not in (3, 50, 60, 61)]
    before = dev.stats()["fallback_queries"]
    (d_, i_), names = logged_launches(dev, lambda: ix.batchSearch(bad, 10))
    assert "list_scan" in names and "query_operands" not in names
    assert 4 <= dev.stats()["fallback_queries"] - before < 50     # (a zero query ties again in its re-run, which counts too)
    assert_topk_parity(d_[keep], i_[keep], rd[keep], ri[keep])
    assert np.all(d_[[3, 50]] == 0.0) and i_[3].tolist() == i_[50].tolist() == list(range(10))
    got, names = logged_launches(dev, lambda: ix.batchSearch(q, 10))
    assert "list_scan" in names and "query_operands" not in names
    assert_topk_parity(*got, rd, ri)


def test_small_batches_that_overflow_rest_together(vsk, dev, cpu_oracle):
    """No single small batch is evidence; a hundred and more of their queries are."""
    rng = np.random.default_rng(22)
    n, d = 30_000, 48
    base = rng.standard_normal(d).astype(np.float32)
    x = np.linspace(0.01, 1.0, n, dtype=np.float32)[:, None] * base + 1e-3 * rng.standard_normal((n, d)).astype(np.float32)
    ix, codes, scale, offset = _quantised(vsk, dev, x)
    rests = []
    for r in range(8):
        q = (base + 0.1 * rng.standard_normal((40, d))).astype(np.float32)
        got, names = logged_launches(dev, lambda: ix.batchSearch(q, 20))
        rests.append("list_scan" not in names)
        assert_topk_parity(*got, *cpu_oracle.sq8_search(oracle.DOT, q, codes, scale, offset, 20))
    assert not rests[0] and all(rests[4:])


def test_a_bounded_wait_of_the_row_lists_runs_out(vsk, cpu_oracle):
    """One CTA's first row tile is never filled: its waits give up after 2^16 polls, the kernel returns, the call answers Timeout
    and the context stays usable."""
    dev = vsk.CUDAAcceleratorStrategy(0).initialize()
    try:
        rng = np.random.default_rng(41)
        ix, codes, scale, offset = _quantised(vsk, dev, rng.standard_normal((40_000, 128)).astype(np.float32))
        q = rng.standard_normal((300, 128)).astype(np.float32)
        dev.set_tuning(wait_limit_log2=16, test_stall_scan=1)
        with pytest.raises(vsk.Timeout):
            ix.batchSearch(q, 10)
        assert dev.tuning()["test_stall_scan"] == 0          # one shot, taken by this kernel
        dev.set_tuning(wait_limit_log2=0)
        _check(cpu_oracle, ix, codes, scale, offset, q, 10)
        ix.close()
    finally:
        dev.close()


def test_decoded_values_are_divided_as_the_decoder_divides(vsk, dev):
    """Queries along one axis: a distance is minus one decoded value, which has to carry the bits of
    (code - offset) / scale, each operation rounded by itself - ordinary scales, powers of two, and scales and offsets beyond
    the range in which the division is done by a reciprocal."""
    rng = np.random.default_rng(77)
    n, d, k = 20_000, 48, 200
    codes = rng.integers(-128, 128, (n, d)).astype(np.int8)
    scale = np.exp(rng.uniform(-8, 8, d)).astype(np.float32)
    offset = (100 * rng.standard_normal(d)).astype(np.float32)
    scale[:6] = [1.0, 0.25, 3.0, 1.0 / 3.0, 2.0, 7.0]
    offset[:6] = [0.0, 5.0, -17.0, 0.5, 1e-18, 128.0]
    ix = vsk.QuantizedFlatIndex(dev, d, vsk.DistanceMetric.dotProduct, scale, offset)
    ix.add(codes)
    q = np.eye(d, dtype=np.float32)
    dist, ids = ix.batchSearch(q, k)
    x = ((codes.astype(np.float32) - offset) / scale).astype(np.float32)
    for j in range(d):
        assert np.array_equal(dist[j], -x[ids[j], j])
        assert np.array_equal(dist[j], np.sort(-x[:, j])[:k])


def test_decoded_values_with_extreme_parameters(vsk, dev):
    rng = np.random.default_rng(78)
    n, d, k = 20_000, 32, 100
    codes = rng.integers(-128, 128, (n, d)).astype(np.int8)
    for s, o in ((1e-13, 3.0), (1e13, 3.0), (0.7, 1e16), (0.7, 1e-16)):
        scale, offset = np.full(d, s, np.float32), np.full(d, o, np.float32)
        ix = vsk.QuantizedFlatIndex(dev, d, vsk.DistanceMetric.dotProduct, scale, offset)
        ix.add(codes)
        dist, ids = ix.batchSearch(np.eye(d, dtype=np.float32), k)
        x = ((codes.astype(np.float32) - offset) / scale).astype(np.float32)
        for j in range(d):
            assert np.array_equal(dist[j], -x[ids[j], j])
        ix.close()
