"""Where a served request's outputs go: page-locked memory (copied behind the
launch), pageable memory (copied after it) and nowhere, in one mix, whole and
in segments.  Outputs equal the oracle's and digests restate them."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gpu = pytest.importorskip("idash2019_2_gb300.gpu")


@pytest.mark.parametrize("segment_outputs,max_inflight", [(0, 8), (7, 8), (7, 1), (1, 3)])
def test_page_locked_pageable_and_no_outputs(oracle, segment_outputs, max_inflight):
    ctx = gpu.Context(0)
    w = gpu.synth_model(seed=5, n_tags=60, n_targets=90, neighbours=4)
    m = gpu.TrlweModel(ctx, w.model, 180, 1024, 1, 1024)
    srv = gpu.Server(m, hbm_budget=1 << 28, max_inflight=max_inflight, segment_outputs=segment_outputs)  # plans m
    rng = np.random.default_rng(segment_outputs)
    reqs, bufs = [], []
    for i in range(12):
        t0, n_indiv = int(rng.integers(0, 80)), int(rng.integers(1, 2100))
        t1 = t0 + int(rng.integers(1, 10))
        in_shape, out_shape, lo = gpu.serve_input_shape(m, n_indiv, t0, t1)
        h_in = rng.integers(0, 2 ** 32, size=in_shape, dtype=np.uint64).astype(np.uint32).view(np.int32)
        n = int(np.prod(out_shape))
        h_out = [None, np.zeros(out_shape, np.int32), None][i % 3]
        if i % 3 == 2:
            bufs.append(ctx.host_alloc(4 * n))  # page-locked
            h_out = np.ctypeslib.as_array(C.cast(bufs[-1].ptr, C.POINTER(C.c_int32)), (n,)).reshape(out_shape)
            h_out[...] = 0
        reqs.append((n_indiv, t0, t1, h_in, h_out, lo))
    try:
        tickets = [srv.submit(n, t0, t1, h_in=h_in, h_out=h_out) for n, t0, t1, h_in, h_out, _ in reqs]
        res = [srv.wait(t) for t in tickets]
        assert srv.stats()["d2h_bytes"] == sum(q[4].nbytes for q in reqs if q[4] is not None)
    finally:
        srv.close()
    for (n_indiv, t0, t1, h_in, h_out, lo), r in zip(reqs, res):
        sub = w.model.slice_outputs(3 * t0, 3 * t1)
        want = []
        for b in range(h_in.shape[0]):
            rows = np.zeros((180, 2048), np.int32)
            rows[lo:lo + h_in.shape[1]] = h_in[b]
            ns = min(1024, n_indiv - 1024 * b)
            want.append(oracle.trlwe_score(sub.term_ptr, sub.term_feat, sub.term_coef, rows, ns, 1, 1024)[0])
        want = np.stack(want)
        if h_out is not None:
            np.testing.assert_array_equal(h_out, want)
        words = np.ascontiguousarray(want).view(np.uint32).ravel()
        assert r["digest"] == ctx.lib.idash_digest_host(words.ctypes.data_as(C.POINTER(C.c_uint32)), words.size, 0)
    ctx.close()
