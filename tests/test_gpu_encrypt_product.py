"""Encryption with binary keys (csrc/encrypt.cu and csrc/key_product.cu) where the
product's persistent loop turns over: more items of 32 rows than SMs, rows that
are 16- and 4-byte aligned, through a row map, one to many regions to a row.
Masks are the documented stream, and b - a*s - m is the reported noise, for
every row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
gpu = pytest.importorskip("idash2019_2_gb300.gpu")


@pytest.fixture(scope="module")
def ctx():
    c = gpu.Context(0)
    yield c
    c.close()


def _product(a, key):
    """a*s mod (X^N + 1, 2^32), exact in 64-bit floats: |sum| <= N * 2^31 < 2^43."""
    N = len(key)
    d = torch.arange(N, device="cuda")[None, :] - torch.arange(N, device="cuda")[:, None]
    k = torch.from_numpy(key).cuda().to(torch.float64)
    toeplitz = torch.where(d >= 0, k[d % N], -k[d % N])
    p = (torch.from_numpy(a).cuda().to(torch.float64) @ toeplitz).to(torch.int64)
    return (p & 0xFFFFFFFF).cpu().numpy().astype(np.uint32)


@pytest.mark.parametrize("N,n_rows,regions,size,ns,shift,mapped", [
    (64, 10001, 1, 64, 64, 0, False), (64, 10001, 4, 15, 14, 4, True), (128, 9777, 128, 1, 1, 0, False),
    (256, 5000, 1, 200, 0, 8, False), (512, 4900, 1, 512, 511, 0, True), (1024, 5100, 10, 102, 100, 0, False),
    (1024, 4897, 1, 1024, 1000, 4, True), (1024, 31, 3, 341, 340, 12, False), (2048, 5000, 2, 1024, 1024, 0, False)])
def test_rows_decrypt_to_their_messages(ctx, oracle, N, n_rows, regions, size, ns, shift, mapped):
    rng = np.random.default_rng(N + n_rows + regions)
    key, seed, n_tags = rng.integers(0, 2, size=N).astype(np.int32), 4242 + N, 17
    geno = rng.integers(-1, 4, size=(n_tags, max(ns, 1))).astype(np.int8)  # -1 and 3: missing
    slot_src = rng.integers(0, 3 * n_tags, size=(n_rows, regions)).astype(np.uint32)
    slot_src[rng.random(slot_src.shape) < 0.1] = 0xFFFFFFFF
    row_out = rng.permutation(n_rows).astype(np.uint32)
    d = {k: torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v).cuda()
         for k, v in (("src", slot_src), ("geno", geno), ("map", row_out))}
    out = torch.full((n_rows * 2 * N + 4,), 77, dtype=torch.int32, device="cuda")
    noise = torch.zeros((n_rows, N), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    params = gpu.encrypt_params(ns, regions, size, N=N)
    gpu.encrypt_device(ctx, params, key, seed, n_rows, d["src"].data_ptr() if ns else 0,
                       d["geno"].data_ptr() if ns else 0, geno.shape[1], out.data_ptr() + shift,
                       gpu.RowLayout(2 * N * 4, 0, -1, -1), d_row_out=d["map"].data_ptr() if mapped else 0,
                       d_noise=noise.data_ptr())
    ctx.sync()
    rows = out.cpu().numpy()[shift // 4:shift // 4 + n_rows * 2 * N].reshape(n_rows, 2 * N)
    if mapped:
        rows = rows[row_out]
    for r in (0, n_rows // 2, n_rows - 1):
        mask = np.array([oracle.lib().oracle_hash32(seed, 21, r * N + j) for j in range(N)], np.uint32)
        np.testing.assert_array_equal(rows[r, :N].view(np.uint32), mask)
    p, v = np.divmod(np.where(slot_src == 0xFFFFFFFF, 0, slot_src).astype(np.int64), 3)
    gv = geno[p][:, :, :ns].astype(np.int64)                                   # [row][region][sample]
    v = v[:, :, None]
    nan = np.array(list(params.nan_t32), np.int64)
    msg = np.where(gv == v, params.one_t32, np.where((gv < 0) | (gv > 2), nan[v], 0))
    msg[slot_src == 0xFFFFFFFF] = 0
    want = np.zeros((n_rows, N), np.uint32)
    for g in range(regions):
        want[:, g * size:g * size + ns] = msg[:, g].astype(np.uint32)
    e = rows[:, N:].view(np.uint32) - _product(np.ascontiguousarray(rows[:, :N]), key) - want
    np.testing.assert_array_equal(e.view(np.int32), noise.cpu().numpy())
