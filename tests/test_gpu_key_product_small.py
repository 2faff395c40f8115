"""The smallest keys that the tensor-core product takes (N = 32, half a chunk of
mask words): decryption word for word against the oracle, encryption through it
(two launches) with b - a*s - m the reported noise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

gpu = pytest.importorskip("idash2019_2_gb300.gpu")

N = 32


@pytest.fixture(scope="module")
def ctx():
    c = gpu.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n_rows,ns,shift", [(1, 32, 0), (31, 1, 4), (33, 16, 0), (64, 17, 8), (10007, 31, 0), (9000, 32, 12)])
def test_decrypt(ctx, oracle, n_rows, ns, shift):
    rng = np.random.default_rng(n_rows + ns)
    rows = rng.integers(0, 2 ** 32, size=(n_rows, 2 * N), dtype=np.uint64).astype(np.uint32).view(np.int32)
    rows[0] = -1
    for key in (rng.integers(0, 2, size=N).astype(np.int32), np.ones(N, np.int32), np.zeros(N, np.int32)):
        d_in, d_out = ctx.device_alloc(rows.nbytes + 64), ctx.device_alloc(n_rows * ns * 4)
        d_in.upload(rows, offset=shift)
        gpu.decrypt_device(ctx, key, d_in.ptr + shift, gpu.RowLayout(2 * N * 4, 0, -1, -1), n_rows, ns, d_out.ptr)
        ctx.sync()
        got, want = d_out.download(dtype=np.float32).reshape(n_rows, ns), oracle.trlwe_decrypt(rows, key, ns)
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
        d_in.free()
        d_out.free()


@pytest.mark.parametrize("n_rows", [1, 45, 8000])
def test_encrypt(ctx, oracle, n_rows):
    rng = np.random.default_rng(n_rows)
    key = rng.integers(0, 2, size=N).astype(np.int32)
    geno = rng.integers(0, 3, size=(5, N)).astype(np.int8)
    src = rng.integers(0, 15, size=n_rows).astype(np.uint32)
    d_src, d_geno = ctx.device_alloc(src.nbytes), ctx.device_alloc(geno.nbytes)
    d_src.upload(src)
    d_geno.upload(geno)
    d_out, d_noise = ctx.device_alloc(n_rows * 2 * N * 4), ctx.device_alloc(n_rows * N * 4)
    params = gpu.encrypt_params(N, 1, N, N=N)
    before = ctx.stats()["kernel_launches"]
    gpu.encrypt_device(ctx, params, key, 5, n_rows, d_src.ptr, d_geno.ptr, N, d_out.ptr,
                       gpu.RowLayout(2 * N * 4, 0, -1, -1), d_noise=d_noise.ptr)
    ctx.sync()
    assert ctx.stats()["kernel_launches"] == before + 2
    rows = d_out.download(dtype=np.int32).reshape(n_rows, 2 * N)
    noise = d_noise.download(dtype=np.int32).reshape(n_rows, N)
    msg = np.where(geno[src // 3].astype(np.uint32) == (src % 3)[:, None], np.uint32(params.one_t32), np.uint32(0))
    product = np.stack([oracle.negacyclic_mul(key, r[:N].view(np.uint32)) for r in rows]).astype(np.uint32)
    np.testing.assert_array_equal((rows[:, N:].view(np.uint32) - product - msg).view(np.int32), noise)
    for b in (d_src, d_geno, d_out, d_noise):
        b.free()
