"""A new model's first pass: plans that are seldom wanted are not timed, where one
that mostly is the fastest works; outputs are the oracle's whichever plan wins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gpu = pytest.importorskip("idash2019_2_gb300.gpu")


@pytest.fixture(scope="module")
def ctx():
    c = gpu.Context(0)
    yield c
    c.close()


# (regions, coefficient scale): coefficients beyond two digits have no tensor-core plan
@pytest.mark.parametrize("regions,scale,most", [(10, 1, 24), (3, 1, 24), (3, 100000, None), (1, 1, None)])
def test_first_pass(ctx, oracle, regions, scale, most):
    size = 1024 // regions
    csr = gpu.synth_model(seed=regions, n_tags=90, n_targets=120, neighbours=6).model
    coef = (csr.term_coef.astype(np.int64) * scale).astype(np.int32)
    csr = gpu.CSRModel(csr.term_ptr, csr.term_feat, coef)
    n_rows = (270 + regions - 1) // regions
    rows = np.random.default_rng(regions).integers(0, 2 ** 32, size=(n_rows, 2048), dtype=np.uint64)
    rows = rows.astype(np.uint32).view(np.int32)
    want, _ = oracle.trlwe_score(csr.term_ptr, csr.term_feat, coef, rows, size, regions, size)
    m = gpu.TrlweModel(ctx, csr, n_rows, size, regions, size)
    d_in, d_out = ctx.device_alloc(rows.nbytes), ctx.device_alloc(csr.n_out * 8192)
    d_in.upload(rows)
    before = ctx.stats()["kernel_launches"]
    for _ in range(2):
        d_out.zero()
        m.score_device(d_in.ptr, gpu.DENSE_TRLWE, d_out.ptr, gpu.DENSE_TRLWE)
        ctx.sync()
        np.testing.assert_array_equal(d_out.download(dtype=np.int32).reshape(csr.n_out, 2048), want)
    if most:  # the tensor-core plan and four windows, four times each, and the two passes
        assert ctx.stats()["kernel_launches"] - before <= most
    m.free()
    d_in.free()
    d_out.free()
