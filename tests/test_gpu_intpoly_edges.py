"""Integer-polynomial scoring where its persistent loop, ring and groups turn
over, bit for bit against the oracle's schoolbook product: more groups than
SMs of one to three outputs, none to 22 terms (a fold after every seventh),
extreme words and coefficients, and weights replaced on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gpu = pytest.importorskip("idash2019_2_gb300.gpu")


@pytest.fixture(scope="module")
def ctx():
    c = gpu.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n_groups,lengths,max_abs", [
    (330, [0, 1, 2], 8192), (40, [6, 7, 8, 14, 15, 22], 8192), (1, [3], 32767), (170, [1], 32767)])
def test_groups_and_folds(ctx, oracle, n_groups, lengths, max_abs):
    rng = np.random.default_rng(n_groups)
    n_rows, ns, rs = 21, 900, 1000
    lists = []
    for g in range(n_groups):
        rows_of = rng.integers(0, n_rows, size=lengths[g % len(lengths)]).astype(np.uint32)
        lists += [rows_of] * (1 + g % 3)
    ptr = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.uint64)
    feat = np.concatenate(lists).astype(np.uint32)
    n_out, n_terms = len(lists), int(ptr[-1])
    poly = rng.choice(np.array([-max_abs, max_abs, -1, 0, max_abs // 3], np.int16), size=(n_terms, 1024))
    other = rng.integers(-max_abs, max_abs + 1, size=(n_terms, 1024)).astype(np.int16)
    rows = rng.choice(np.array([-2 ** 31, 2 ** 31 - 1, -2 ** 31 + 1, 0, 123456789], np.int32), size=(n_rows, 2048))
    rows[::2] = rng.integers(0, 2 ** 32, size=rows[::2].shape, dtype=np.uint64).astype(np.uint32).view(np.int32)
    bias = rng.integers(-8192, 8192, size=n_out).astype(np.int32)
    m = gpu.IntpolyModel(ctx, gpu.CSRModel(ptr, feat, np.zeros(n_terms, np.int32)), poly, n_rows, ns, rs, bias=bias,
                         max_abs_coef=max_abs)
    d_in, d_out = ctx.device_alloc(rows.nbytes), ctx.device_alloc(n_out * 8192)
    d_in.upload(rows)
    d_poly = ctx.device_alloc(max(other.nbytes, 16))
    d_poly.upload(other)
    for step, weights in enumerate((poly, other)):
        if step:
            m.set_weights(d_poly.ptr)
        d_out.zero()
        m.score_device(d_in.ptr, gpu.DENSE_TRLWE, 0, n_out, d_out.ptr, gpu.DENSE_TRLWE)
        ctx.sync()
        want = oracle.intpoly_score(ptr, feat, weights, bias, rows, ns, rs, 0, n_out)
        np.testing.assert_array_equal(d_out.download(dtype=np.int32).reshape(n_out, 2048), want)
    m.free()
    for d in (d_in, d_out, d_poly):
        d.free()
