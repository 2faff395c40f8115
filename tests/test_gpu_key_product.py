"""The tensor-core product of masks with a binary key (csrc/key_product.cu)
behind decryption, word for word against the oracle at the edges of its tiles:
rows per item, columns per load, step and pair of tiles, more row tiles than
SMs, rows that are only 4-byte aligned, and the largest digit sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gpu = pytest.importorskip("idash2019_2_gb300.gpu")


@pytest.fixture(scope="module")
def ctx():
    c = gpu.Context(0)
    yield c
    c.close()


def _check(ctx, oracle, rows, key, ns, shift=0):
    n_rows, N = rows.shape[0], rows.shape[1] // 2
    d_in = ctx.device_alloc(rows.nbytes + 64)
    d_in.upload(rows, offset=shift)
    d_out = ctx.device_alloc(n_rows * ns * 4)
    gpu.decrypt_device(ctx, key, d_in.ptr + shift, gpu.RowLayout(2 * N * 4, 0, -1, -1), n_rows, ns, d_out.ptr)
    ctx.sync()
    got = d_out.download(dtype=np.float32).reshape(n_rows, ns)
    want = oracle.trlwe_decrypt(rows, key, ns)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
    d_in.free()
    d_out.free()


@pytest.mark.parametrize("N,n_rows,ns,shift", [
    (64, 1, 64, 0), (128, 41, 33, 0), (512, 80, 47, 4), (1024, 39, 48, 0), (1024, 40, 49, 8), (1024, 1, 513, 0),
    (1024, 32, 257, 0), (1024, 33, 31, 0), (512, 31, 512, 0), (2048, 64, 769, 0), (64, 5000, 3, 4),
    (1024, 6121, 100, 0), (1024, 3200, 1000, 4), (2048, 83, 2048, 0), (2048, 1, 1025, 12)])
def test_tile_edges(ctx, oracle, N, n_rows, ns, shift):
    rng = np.random.default_rng(N + n_rows + ns)
    rows = rng.integers(0, 2 ** 32, size=(n_rows, 2 * N), dtype=np.uint64).astype(np.uint32).view(np.int32)
    _check(ctx, oracle, rows, rng.integers(0, 2, size=N).astype(np.int32), ns, shift)


@pytest.mark.parametrize("word", [-1, 0x7FF, 0x3FF800, -0x400000, -2 ** 31])
def test_largest_sums(ctx, oracle, word):
    """Every key bit set and every mask word with full digits: N * 2047 per digit at N = 2048."""
    rows = np.full((45, 4096), word, np.int32)
    _check(ctx, oracle, rows, np.ones(2048, np.int32), 2048)
