"""One integer-polynomial model used from several streams: its calls share the
resident weights and the buffer of transformed inputs, and take effect in the
order they are made, also captured into a graph.  Bit for bit against the
oracle's schoolbook product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
gpu = pytest.importorskip("idash2019_2_gb300.gpu")

N_ROWS, N_OUT, TERMS = 300, 6, 9


@pytest.fixture(scope="module")
def case(oracle):
    rng = np.random.default_rng(3)
    ctx = gpu.Context(0)
    ptr = np.arange(N_OUT + 1, dtype=np.uint64) * TERMS
    feat = rng.integers(0, N_ROWS, size=N_OUT * TERMS).astype(np.uint32)
    weights = [rng.integers(-8192, 8192, size=(len(feat), 1024)).astype(np.int16) for _ in range(2)]
    rows = [rng.integers(0, 2 ** 32, size=(N_ROWS, 2048), dtype=np.uint64).astype(np.uint32).view(np.int32)
            for _ in range(2)]
    bias = np.zeros(N_OUT, np.int32)
    want = [[oracle.intpoly_score(ptr, feat, w, bias, x, 1024, 1024, 0, N_OUT) for x in rows] for w in weights]
    m = gpu.IntpolyModel(ctx, gpu.CSRModel(ptr, feat, np.zeros(len(feat), np.int32)), weights[0], N_ROWS, 1024, 1024)
    yield (m, [torch.from_numpy(x).cuda() for x in rows], [torch.from_numpy(w).cuda() for w in weights], want)
    m.free()
    ctx.close()


def _score(m, x, y, stream):
    m.score_device(x.data_ptr(), gpu.DENSE_TRLWE, 0, N_OUT, y.data_ptr(), gpu.DENSE_TRLWE, stream=stream.cuda_stream)


def test_two_streams(case):
    m, x, w, want = case
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    y = [torch.zeros((N_OUT, 2048), dtype=torch.int32, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    for _ in range(10):
        _score(m, x[0], y[0], a)
        _score(m, x[1], y[1], b)
        m.set_weights(w[1].data_ptr(), stream=b.cuda_stream)
        _score(m, x[0], y[2], a)
        _score(m, x[1], y[3], b)
        m.set_weights(w[0].data_ptr(), stream=a.cuda_stream)
    torch.cuda.synchronize()
    for got, exp in zip(y, (want[0][0], want[0][1], want[1][0], want[1][1])):
        np.testing.assert_array_equal(got.cpu().numpy(), exp)


def test_captured(case):
    m, x, w, want = case
    y = [torch.zeros((N_OUT, 2048), dtype=torch.int32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    _score(m, x[0], y[0], torch.cuda.current_stream())  # the model's buffers are there from now on
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _score(m, x[0], y[0], torch.cuda.current_stream())
    b = torch.cuda.Stream()
    for k in (1, 0, 1, 0):
        m.set_weights(w[k].data_ptr(), stream=b.cuda_stream)
        g.replay()
        _score(m, x[1], y[1], b)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(y[0].cpu().numpy(), want[k][0])
        np.testing.assert_array_equal(y[1].cpu().numpy(), want[k][1])
