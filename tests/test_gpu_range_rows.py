"""Ranges of models with several regions to a row: a request brings the rows that
its own outputs read, no more, whatever plan the model has and however its
blocks are cut.  Outputs word for word against the oracle; a window that lacks
a row is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gpu = pytest.importorskip("idash2019_2_gb300.gpu")

TC_KIND = 4


@pytest.fixture(scope="module")
def ctx():
    c = gpu.Context(0)
    yield c
    c.close()




@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("regions,size", [(2, 512), (3, 341), (10, 102), (40, 25)])
@pytest.mark.parametrize("neighbours,shuffled", [(4, False), (25, False), (4, True)])
def test_a_range_brings_its_own_rows(ctx, oracle, regions, size, neighbours, shuffled, tuned):
    tags, targets, ns = 260, 300, size - 1
    csr = gpu.synth_model(seed=regions + neighbours, n_tags=tags, n_targets=targets, neighbours=neighbours).model
    n_rows = (3 * tags + regions - 1) // regions
    rng = np.random.default_rng(regions)
    rows = rng.integers(0, 2 ** 32, size=(n_rows, 2048), dtype=np.uint64).astype(np.uint32).view(np.int32)
    perm = rng.permutation(n_rows).astype(np.uint32) if shuffled else np.arange(n_rows, dtype=np.uint32)
    stored = np.empty_like(rows)
    stored[perm] = rows  # FeatIndex i is at input row perm[i]
    m = gpu.TrlweModel(ctx, csr, n_rows, ns, regions, size, row_of_index=perm)
    want, _ = oracle.trlwe_score(csr.term_ptr, csr.term_feat, csr.term_coef, rows, ns, regions, size)
    if tuned:
        d_in, d_out = ctx.device_alloc(rows.nbytes), ctx.device_alloc(csr.n_out * 8192)
        d_in.upload(stored)
        m.score_device(d_in.ptr, gpu.DENSE_TRLWE, d_out.ptr, gpu.DENSE_TRLWE)
        ctx.sync()
        d_in.free()
        d_out.free()
    for lo, hi in [(0, 1), (1, 4), (126, 131), (383, 384), (300, 700), (csr.n_out - 2, csr.n_out), (0, csr.n_out)]:
        f = csr.term_feat[int(csr.term_ptr[lo]):int(csr.term_ptr[hi])]
        read = perm[f[f != 0xFFFFFFFF] // regions]
        own = (int(read.min()), int(read.max()) + 1)
        a, b = m.input_rows(lo, hi)
        assert a <= own[0] and own[1] <= b
        if m.info()["kernel"] == TC_KIND:
            assert (a, b) == own
        for base, end in {(a, b), (max(0, a - 3), min(n_rows, b + 2))}:
            d_in, d_out = ctx.device_alloc((end - base) * 8192), ctx.device_alloc((hi - lo) * 8192)
            d_in.upload(stored[base:end])
            d_out.zero()
            m.score_range(lo, hi, 0, d_in.ptr, gpu.DENSE_TRLWE, base, end - base, d_out.ptr, gpu.DENSE_TRLWE)
            ctx.sync()
            np.testing.assert_array_equal(d_out.download(dtype=np.int32).reshape(hi - lo, 2048), want[lo:hi])
            with pytest.raises(gpu.IdashError) as e:
                m.score_range(lo, hi, 0, d_in.ptr, gpu.DENSE_TRLWE, own[0] + 1, end - base, d_out.ptr, gpu.DENSE_TRLWE)
            assert e.value.name == "IDASH_ERR_INDEX"
            d_in.free()
            d_out.free()
    m.free()


def test_outputs_without_terms_bring_no_row(ctx, oracle):
    """Constants only, in a block whose other outputs read rows; and a feature
    whose coefficients cancel."""
    regions, size, ns = 4, 256, 200
    ptr = np.array([0, 2, 3, 3, 6], np.uint64)
    feat = np.array([9, 0xFFFFFFFF, 0xFFFFFFFF, 13, 14, 14], np.uint32)
    coef = np.array([5, 3, -7, 100, 8, -8], np.int32)
    csr = gpu.CSRModel(ptr, feat, coef)
    rows = np.random.default_rng(1).integers(0, 2 ** 32, size=(4, 2048), dtype=np.uint64).astype(np.uint32).view(np.int32)
    want, _ = oracle.trlwe_score(ptr, feat, coef, rows, ns, regions, size)
    m = gpu.TrlweModel(ctx, csr, 4, ns, regions, size)
    d_in, d_out = ctx.device_alloc(16), ctx.device_alloc(2 * 8192)
    d_out.zero()
    a, b = m.input_rows(1, 3)
    if m.info()["kernel"] == TC_KIND:
        assert (a, b) == (0, 0)
        m.score_range(1, 3, 0, d_in.ptr, gpu.DENSE_TRLWE, 0, 0, d_out.ptr, gpu.DENSE_TRLWE)
        ctx.sync()
        np.testing.assert_array_equal(d_out.download(dtype=np.int32).reshape(2, 2048), want[1:3])
    m.free()
    d_in.free()
    d_out.free()


@pytest.mark.parametrize("regions,size,kernel", [(1, 1024, 0), (1, 1024, 2), (3, 341, 0)])
def test_variances_of_terms_that_cancel(ctx, oracle, regions, size, kernel):
    """A feature whose coefficients cancel is read for its variance alone: a window
    without its row is refused where variances are asked for, and taken where not."""
    far = 3 * 50 if regions > 1 else 50  # region 0 of row 50
    ptr, ns = np.array([0, 4, 5], np.uint64), size - 1
    feat = np.array([0, regions, far, far, regions], np.uint32)
    coef = np.array([3, 4, 7, -7, 2], np.int32)
    n_rows = 60
    rows = np.random.default_rng(2).integers(0, 2 ** 32, size=(n_rows, 2048), dtype=np.uint64).astype(np.uint32).view(np.int32)
    var = np.arange(1.0, n_rows + 1.0)
    rec = np.zeros((n_rows, gpu.RECORD_BYTES), np.uint8)
    rec[:, 8:8200] = rows.view(np.uint8).reshape(n_rows, 8192)
    rec[:, 8200:] = var[:, None].view(np.uint8)
    want, _ = oracle.trlwe_score(ptr, feat, coef, rows, ns, regions, size)
    ctx.set_option("kernel", kernel)
    try:
        m = gpu.TrlweModel(ctx, gpu.CSRModel(ptr, feat, coef), n_rows, ns, regions, size)
    finally:
        ctx.set_option("kernel", 0)
    assert m.input_rows(0, 1) == (0, 51)
    d_in, d_out = ctx.device_alloc(rec.nbytes + 16), ctx.device_alloc(2 * gpu.RECORD_BYTES + 16)
    d_in.upload(rec, offset=8)
    d_out.zero()
    at = (d_in.ptr + 8, gpu.RECORD_IN, 0)
    m.score_range(0, 1, 0, *at, 51, d_out.ptr + 8, gpu.RECORD_OUT)
    ctx.sync()
    got = d_out.download(nbytes=gpu.RECORD_BYTES, offset=8)
    np.testing.assert_array_equal(got[8:8200].view(np.int32), want[0])
    assert got[8200:].view(np.float64)[0] == 9 * 1.0 + 16 * 2.0 + 49 * 51.0 + 49 * 51.0
    with pytest.raises(gpu.IdashError) as e:
        m.score_range(0, 1, 0, *at, 2, d_out.ptr + 8, gpu.RECORD_OUT)
    assert e.value.name == "IDASH_ERR_INDEX"
    m.score_range(0, 1, 0, *at, 2, d_out.ptr, gpu.DENSE_TRLWE)
    ctx.sync()
    np.testing.assert_array_equal(d_out.download(nbytes=8192, dtype=np.int32), want[0])
    m.free()
    d_in.free()
    d_out.free()
