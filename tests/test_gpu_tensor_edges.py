"""The tensor-core scoring kernel's branches at their edges, word for word
against the oracle: rows that are consecutive, partly and wholly scattered (one
and two producers), every set of buffers (padded K up to 64, 80, 96 and 192),
outputs in order and through a row map, blocks that are not full, and LWE rows
that end inside a 32-column box with samples shorter than it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gpu = pytest.importorskip("idash2019_2_gb300.gpu")

TC_KIND = 4


@pytest.fixture(scope="module")
def ctx():
    c = gpu.Context(0)
    c.set_option("kernel", 5)
    yield c
    c.set_option("kernel", 0)
    c.close()


def _model(rng, n_out, k, n_rows, scatter):
    """Blocks of 128 outputs over the same k rows; a row is left out at each
    output.  scatter: the share of the rows that lie apart."""
    ptr, feat, coef = [0], [], []
    for o in range(n_out):
        if o % 128 == 0:
            rows = np.arange(k) + rng.integers(0, n_rows - k + 1)
            away = rng.random(k) < scatter
            rows[away] = rng.choice(np.setdiff1d(np.arange(n_rows), rows), size=int(away.sum()), replace=False)
        take = np.delete(rows, o % k) if k > 1 else rows
        feat += [int(r) for r in take]
        coef += [int(c) for c in rng.integers(-8000, 8000, size=len(take))]
        if o % 3 == 0:
            feat.append(0xFFFFFFFF)
            coef.append(int(rng.integers(-2 ** 31, 2 ** 31)))
        ptr.append(len(feat))
    return gpu.CSRModel(np.array(ptr, np.uint64), np.array(feat, np.uint32), np.array(coef, np.int64).astype(np.int32))


def _words(rng, shape):
    return rng.integers(0, 2 ** 32, size=shape, dtype=np.uint64).astype(np.uint32).view(np.int32)


@pytest.mark.parametrize("scatter", [0.0, 0.01, 1.0])
@pytest.mark.parametrize("k", [1, 15, 33, 64, 65, 80, 81, 96, 97, 192])
def test_trlwe(ctx, oracle, k, scatter):
    rng = np.random.default_rng(1000 * k + int(100 * scatter))
    n_out, n_rows, ns = 128 + (33 if k % 2 else 1), 420, 700
    csr = _model(rng, n_out, k, n_rows, scatter)
    rows = _words(rng, (n_rows, 2048))
    want, _ = oracle.trlwe_score(csr.term_ptr, csr.term_feat, csr.term_coef, rows, ns, 1, 1024)
    m = gpu.TrlweModel(ctx, csr, n_rows, ns, 1, 1024)
    assert m.info()["kernel"] == TC_KIND
    d_in, d_out = ctx.device_alloc(rows.nbytes), ctx.device_alloc(n_out * 8192)
    d_in.upload(rows)
    m.score_device(d_in.ptr, gpu.DENSE_TRLWE, d_out.ptr, gpu.DENSE_TRLWE)
    ctx.sync()
    np.testing.assert_array_equal(d_out.download(dtype=np.int32).reshape(n_out, 2048), want)
    lo, hi = 3, n_out - 1
    d_out.zero()
    m.score_range(lo, hi, 0, d_in.ptr, gpu.DENSE_TRLWE, 0, n_rows, d_out.ptr, gpu.DENSE_TRLWE)
    ctx.sync()
    np.testing.assert_array_equal(d_out.download(dtype=np.int32).reshape(n_out, 2048)[:hi - lo], want[lo:hi])
    m.free()
    d_in.free()
    d_out.free()


@pytest.mark.parametrize("n,n_indiv", [(1, 30), (7, 9), (30, 3), (31, 5), (32, 1), (63, 1), (64, 2), (630, 3)])
@pytest.mark.parametrize("k,scatter", [(20, 0.0), (20, 1.0), (120, 1.0)])
def test_lwe(ctx, oracle, n, n_indiv, k, scatter):
    rng = np.random.default_rng(n * 100 + n_indiv + k)
    n_out, n_rows = 131, 300
    csr = _model(rng, n_out, k, n_rows, scatter)
    stride, words = gpu.lwe_row_words(n_indiv, n), n_indiv * (n + 1)
    rows = np.zeros((n_rows, stride), np.int32)
    rows[:, :words] = _words(rng, (n_rows, words))
    d_in, d_out = ctx.device_alloc(rows.nbytes), ctx.device_alloc(n_out * stride * 4)
    d_in.upload(rows)
    d_out.zero()
    m = gpu.LweModel(ctx, csr, n_rows, n_indiv, n)
    m.score_device(n_indiv, d_in.ptr, stride, 0, n_out, d_out.ptr, stride)
    ctx.sync()
    assert m.info()["kernel"] == TC_KIND
    got = d_out.download(dtype=np.int32).reshape(n_out, stride)
    want = oracle.lwe_score(csr.term_ptr, csr.term_feat, csr.term_coef, np.ascontiguousarray(rows[:, :words]),
                            n_indiv, 0, n_out, n=n)
    np.testing.assert_array_equal(got[:, :words], want)
    assert not got[:, words:].any()
    m.free()
    d_in.free()
    d_out.free()


@pytest.mark.parametrize("regions,size,ns", [
    (1, 800, 799), (2, 512, 512), (3, 341, 300), (3, 340, 1), (7, 146, 100), (10, 102, 101), (16, 64, 64), (40, 25, 25),
    (341, 3, 2), (1024, 1, 1)])
@pytest.mark.parametrize("tags,targets,neighbours", [(60, 90, 1), (130, 100, 5), (100, 45, 25)])
def test_rotated_rows(ctx, oracle, regions, size, ns, tags, targets, neighbours):
    """Several regions to a row: rotations that keep 16, 8 and 4 bytes aligned,
    tiles before, at and after a polynomial's end, and columns that are zeros;
    dense outputs, a range of them, and records through a row map."""
    w = gpu.synth_model(seed=regions + neighbours, n_tags=tags, n_targets=targets, neighbours=neighbours)
    csr, n_rows = w.model, (3 * tags + regions - 1) // regions
    rng = np.random.default_rng(regions)
    rows = _words(rng, (n_rows, 2048))
    rows[0, ::3] = -2 ** 31
    want, _ = oracle.trlwe_score(csr.term_ptr, csr.term_feat, csr.term_coef, rows, ns, regions, size)
    m = gpu.TrlweModel(ctx, csr, n_rows, ns, regions, size)
    assert m.info()["kernel"] == TC_KIND
    d_in, d_out = ctx.device_alloc(rows.nbytes), ctx.device_alloc(m.n_out * gpu.RECORD_BYTES + 16)
    d_in.upload(rows)
    for graph in (1, 0):
        ctx.set_option("graph", graph)
        d_out.upload(np.full(m.n_out * 2048, 77, np.int32))
        m.score_device(d_in.ptr, gpu.DENSE_TRLWE, d_out.ptr, gpu.DENSE_TRLWE)
        ctx.sync()
        got = d_out.download(nbytes=m.n_out * 8192, dtype=np.int32).reshape(m.n_out, 2048)
        np.testing.assert_array_equal(got, want)
    ctx.set_option("graph", 1)
    lo, hi = 2, m.n_out - 3
    d_out.upload(np.full(m.n_out * 2048, 77, np.int32))
    m.score_range(lo, hi, 0, d_in.ptr, gpu.DENSE_TRLWE, 0, n_rows, d_out.ptr, gpu.DENSE_TRLWE)
    ctx.sync()
    got = d_out.download(nbytes=m.n_out * 8192, dtype=np.int32).reshape(m.n_out, 2048)
    np.testing.assert_array_equal(got[:hi - lo], want[lo:hi])
    assert (got[hi - lo:] == 77).all()
    m.free()
    out_row = rng.permutation(csr.n_out).astype(np.uint32)
    m = gpu.TrlweModel(ctx, csr, n_rows, ns, regions, size, out_row=out_row)
    m.score_device(d_in.ptr, gpu.DENSE_TRLWE, d_out.ptr + 8, gpu.RECORD_OUT)
    ctx.sync()
    got = d_out.download(nbytes=m.n_out * gpu.RECORD_BYTES, offset=8, dtype=np.int32).reshape(m.n_out, -1)
    np.testing.assert_array_equal(got[out_row, 2:2050], want)
    m.free()
    d_in.free()
    d_out.free()
