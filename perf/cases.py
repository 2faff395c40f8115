"""Timed workloads of the library, each through the entry points a program calls.

A case is one pass of one of these kinds:

  trlwe     score a resident TRLWE-packed model on device rows (the cloud step)
  records   the same on the files' record images: FeatIndex -> row map, output
            permutation, headers and variances (what idash_cloud does)
  range     one request's contiguous targets from a resident model
  lwe       score a resident per-individual LWE model on device rows
  intpoly   score a resident integer-polynomial model on device rows
  reweight  replace an integer-polynomial model's weights, then score
  encrypt   party A: fresh TRLWE encryptions of one-hot genotypes
  decrypt   party A: phases of output TRLWE as float scores
  serve     an online server: a burst of requests with host payloads

Shapes follow the benchmark's workloads (bench.py) and the reference's test
set: 1,000-odd individuals, thousands of tag SNPs, five targets per tag, 5 to
50 neighbours.
"""
import numpy as np
import torch

from idash2019_2_gb300 import gpu

N = 1024
CONSTANT = 0xFFFFFFFF
UNEVEN = [5, 10, 20, 30, 50]

_ctx = None


def _context():
    """The process's one GPU context, as a program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = gpu.Context(0)
    return _ctx


def listed():
    return [
        # A hundred individuals, ten regions packed per ciphertext (the
        # reference's own packing of a small panel): the launch-bound end.
        {"name": "trlwe_small", "kind": "trlwe", "samples": 100, "tags": 500, "targets": 2000, "neighbours": 5},
        # The whole challenge test set in the reference's layout: the headline.
        {"name": "trlwe_full", "kind": "trlwe", "samples": 1000, "tags": 16184, "targets": 80882, "neighbours": 5},
        # A chromosome part as idash_cloud scores it from its files.
        {"name": "records_odd", "kind": "records", "samples": 1004, "tags": 5003, "targets": 30007, "neighbours": 10},
        # One user's request of a few targets against a resident model.
        {"name": "range_tiny", "kind": "range", "samples": 517, "tags": 1618, "targets": 8088, "neighbours": 5,
         "first": 3001, "count": 50},
        # The small panel in the per-individual layout.
        {"name": "lwe_small", "kind": "lwe", "indiv": 100, "n": 1024, "tags": 500, "targets": 2000, "neighbours": 5},
        # Neighbourhoods of 5 to 50 tags, 1,000 individuals: the heavy arithmetic.
        {"name": "lwe_uneven", "kind": "lwe", "indiv": 1000, "n": 1024, "tags": 200, "targets": 1000,
         "neighbours": 0},
        # Another key size and a ragged row (37 samples of 631 words).
        {"name": "lwe_odd", "kind": "lwe", "indiv": 37, "n": 630, "tags": 1009, "targets": 3001, "neighbours": 7},
        # Dense integer-polynomial weights, 60 terms per output.
        {"name": "intpoly", "kind": "intpoly", "tags": 600, "targets": 3000, "neighbours": 20},
        # A model update: new weights, then a pass with them.
        {"name": "reweight", "kind": "reweight", "tags": 101, "targets": 503, "neighbours": 20},
        # Party A encrypts the test set's 48,552 input ciphertexts.
        {"name": "encrypt_full", "kind": "encrypt", "samples": 1000, "tags": 16184},
        # Party A decrypts every output of the test set.
        {"name": "decrypt_full", "kind": "decrypt", "samples": 1000, "rows": 242646},
        # A burst of small requests to the server, ciphertexts from and to host memory.
        {"name": "serve_burst", "kind": "serve", "tags": 1618, "targets": 8088, "neighbours": 10, "requests": 16,
         "count": 203},
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], evenly over the logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["trlwe", "records", "range", "lwe", "intpoly", "reweight", "encrypt", "decrypt", "serve"])
    case = {"kind": kind}
    neighbours = _spread(rng, 3, 30)
    if kind in ("trlwe", "records"):
        tags = _spread(rng, 64, 8000)
        case.update(samples=_spread(rng, 60, 1024), tags=tags, targets=_spread(rng, 50, 24000), neighbours=neighbours)
    elif kind == "range":
        tags = _spread(rng, 200, 4000)
        targets = 5 * tags
        count = _spread(rng, 10, targets // 2)
        case.update(samples=rng.randint(513, 1024), tags=tags, targets=targets, neighbours=neighbours,
                    first=rng.randint(0, targets - count), count=count)
    elif kind == "lwe":
        indiv, n = _spread(rng, 1, 1000), rng.choice([500, 630, 1024])
        # at most 6 GB of outputs
        most = max(10, min(5000, 6 * 10 ** 9 // (3 * 4 * indiv * (n + 1))))
        tags = _spread(rng, 60, 400)
        case.update(indiv=indiv, n=n, tags=tags, targets=_spread(rng, 10, most),
                    neighbours=rng.choice([0, neighbours]))
    elif kind in ("intpoly", "reweight"):
        neighbours = _spread(rng, 2, 40)
        terms = 3 * 3 * neighbours  # per target
        most = (500000 if kind == "intpoly" else 90000) // terms
        case.update(tags=_spread(rng, 60, 1500), targets=_spread(rng, 20, max(21, most)), neighbours=neighbours)
    elif kind == "encrypt":
        case.update(samples=_spread(rng, 60, 1024), tags=_spread(rng, 20, 16000))
    elif kind == "decrypt":
        case.update(samples=_spread(rng, 40, 1024), rows=_spread(rng, 30, 200000))
    else:
        tags = _spread(rng, 300, 2000)
        case.update(tags=tags, targets=5 * tags, neighbours=neighbours, requests=rng.randint(1, 24),
                    count=_spread(rng, 5, 300))
    return case


def _packing(samples):
    """(NUM_REGIONS, REGION_SIZE) for this many individuals, as the reference packs them."""
    regions = max(1, N // samples)
    return regions, N // regions


def _model(case, seed):
    k = case["neighbours"]
    return gpu.synth_model(seed, case["tags"], case["targets"], neighbours=k, choices=None if k else UNEVEN).model


def _words(seed, *shape):
    """Uniform 32-bit words (what ciphertexts look like) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-2 ** 31, 2 ** 31, shape, generator=g, device="cuda", dtype=torch.int32)


def _empty_rows(n, words):
    return torch.zeros((n, words), dtype=torch.int32, device="cuda")


class _State:
    """What a program holds between passes."""

    def __init__(self, case, **kv):
        self.case, self.ctx = case, _context()
        self.__dict__.update(kv)

    def __del__(self):
        server = self.__dict__.get("server")
        if server is not None:
            server.close()  # before the model it runs on


def _prepare_trlwe(case, seed):
    csr = _model(case, seed)
    regions, rs = _packing(case["samples"])
    n_rows = (3 * case["tags"] + regions - 1) // regions
    m = gpu.TrlweModel(_context(), csr, n_rows, case["samples"], regions, rs)
    return _State(case, csr=csr, model=m, regions=regions, rs=rs, rows=_words(seed, n_rows, 2 * N),
                  out=_empty_rows(csr.n_out, 2 * N))


def _prepare_records(case, seed):
    csr = _model(case, seed)
    regions, rs = _packing(case["samples"])
    n_rows = (3 * case["tags"] + regions - 1) // regions
    rng = np.random.default_rng(seed)
    words = gpu.RECORD_BYTES // 4
    # the payload starts 8 bytes into a record: shift the image by 8 bytes so that it is 16-byte aligned
    image = _words(seed, n_rows * words + 4)
    var = torch.full((n_rows,), 2.0 ** -50, dtype=torch.float64, device="cuda")
    image[2:-2].view(n_rows, words)[:, words - 2:] = var.view(torch.int32).view(n_rows, 2)
    m = gpu.TrlweModel(_context(), csr, n_rows, case["samples"], regions, rs,
                       out_index=rng.permutation(csr.n_out).astype(np.uint32) * 3 + 7,
                       out_row=rng.permutation(csr.n_out).astype(np.uint32),
                       row_of_index=rng.permutation(n_rows).astype(np.uint32))
    out = torch.zeros(csr.n_out * words + 4, dtype=torch.int32, device="cuda")
    return _State(case, csr=csr, model=m, image=image, out=out)


def _prepare_range(case, seed):
    s = _prepare_trlwe(case, seed)
    lo, hi = 3 * case["first"], 3 * (case["first"] + case["count"])
    row_lo, row_hi = s.model.input_rows(lo, hi)
    s.lo, s.hi, s.row_lo, s.n_rows = lo, hi, row_lo, row_hi - row_lo
    s.rows = s.rows[row_lo:row_hi].clone()  # the request brings only the rows it reads
    s.out = _empty_rows(hi - lo, 2 * N)
    return s


def _prepare_lwe(case, seed):
    csr = _model(case, seed)
    stride = gpu.lwe_row_words(case["indiv"], case["n"])
    m = gpu.LweModel(_context(), csr, 3 * case["tags"], case["indiv"], case["n"])
    return _State(case, csr=csr, model=m, stride=stride, rows=_words(seed, 3 * case["tags"], stride),
                  out=_empty_rows(csr.n_out, stride))


def _prepare_intpoly(case, seed):
    ctx = _context()
    csr = _model(case, seed)
    const = csr.term_feat == CONSTANT
    owner = np.repeat(np.arange(csr.n_out), np.diff(csr.term_ptr.astype(np.int64)))
    bias = np.zeros(csr.n_out, np.int32)
    bias[owner[const]] = csr.term_coef[const]
    feat = csr.term_feat[~const]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(owner[~const], minlength=csr.n_out))]).astype(np.uint64)
    terms = gpu.CSRModel(ptr, feat, np.zeros(len(feat), np.int32))
    g = torch.Generator(device="cuda").manual_seed(seed)
    polys = torch.randint(-8192, 8192, (len(feat), N), generator=g, device="cuda", dtype=torch.int16)
    torch.cuda.synchronize()
    m = gpu.IntpolyModel(ctx, terms, polys.data_ptr(), 3 * case["tags"], N, N, bias=bias, poly_on_device=True)
    s = _State(case, csr=terms, bias=bias, model=m, rows=_words(seed + 1, 3 * case["tags"], 2 * N),
               out=_empty_rows(csr.n_out, 2 * N))
    if case["kind"] == "reweight":
        s.polys = torch.randint(-8192, 8192, (len(feat), N), generator=g, device="cuda", dtype=torch.int16)
    return s


def _prepare_encrypt(case, seed):
    regions, rs = _packing(case["samples"])
    n_rows = (3 * case["tags"] + regions - 1) // regions
    src = torch.arange(n_rows * regions, dtype=torch.int64, device="cuda")
    src[src >= 3 * case["tags"]] = -1  # no feature in this slot
    g = torch.Generator(device="cuda").manual_seed(seed)
    geno = torch.randint(0, 3, (case["tags"], case["samples"]), generator=g, device="cuda", dtype=torch.int8)
    missing = torch.rand(geno.shape, generator=g, device="cuda") < 0.01
    geno[missing] = -1
    words = gpu.RECORD_BYTES // 4
    return _State(case, params=gpu.encrypt_params(case["samples"], regions, rs), key=gpu.synth_key(seed), seed=seed,
                  n_rows=n_rows, src=src.to(torch.int32), geno=geno,
                  out=torch.zeros(n_rows * words + 4, dtype=torch.int32, device="cuda"))


def _prepare_decrypt(case, seed):
    # scores of 14-bit weights over many tags fill the torus: so do the phases here
    return _State(case, key=gpu.synth_key(seed), rows=_words(seed, case["rows"], 2 * N),
                  out=torch.zeros((case["rows"], case["samples"]), dtype=torch.float32, device="cuda"))


def _prepare_serve(case, seed):
    ctx = _context()
    csr = _model(case, seed)
    ctx.set_option("kernel", 4)  # the server's kernel
    try:
        m = gpu.TrlweModel(ctx, csr, 3 * case["tags"], N, 1, N)
    finally:
        ctx.set_option("kernel", 0)
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(1).integers(1, 2001, case["requests"])  # the same for every seed
    requests = []
    for indiv in sizes.tolist():
        first = int(rng.integers(0, case["targets"] - case["count"]))
        shape_in, shape_out, _ = gpu.serve_input_shape(m, indiv, first, first + case["count"])
        # page-locked arrays that live as long as anything refers to them
        h_in, h_out = (torch.zeros(shape, dtype=torch.int32, pin_memory=True).numpy()
                       for shape in (shape_in, shape_out))
        h_in[...] = rng.integers(-2 ** 31, 2 ** 31, shape_in, dtype=np.int32)
        requests.append((indiv, first, h_in, h_out))
    s = _State(case, csr=csr, model=m, requests=requests)
    s.server = gpu.Server(m, 4 << 30, 64)
    return s


def prepare(case, seed):
    kind = case["kind"]
    make = _prepare_intpoly if kind == "reweight" else globals()["_prepare_" + kind]
    s = make(case, seed)
    torch.cuda.synchronize()
    return s


def run(s):
    kind, case = s.case["kind"], s.case
    dense = gpu.DENSE_TRLWE
    if kind == "trlwe":
        s.model.score_device(s.rows.data_ptr(), dense, s.out.data_ptr(), dense)
    elif kind == "records":
        s.model.score_device(s.image.data_ptr() + 8, gpu.RECORD_IN, s.out.data_ptr() + 8, gpu.RECORD_OUT)
    elif kind == "range":
        s.model.score_range(s.lo, s.hi, case["samples"], s.rows.data_ptr(), dense, s.row_lo, s.n_rows,
                            s.out.data_ptr(), dense)
    elif kind == "lwe":
        s.model.score_device(case["indiv"], s.rows.data_ptr(), s.stride, 0, s.csr.n_out, s.out.data_ptr(), s.stride)
    elif kind in ("intpoly", "reweight"):
        if kind == "reweight":
            s.model.set_weights(s.polys.data_ptr())
        s.model.score_device(s.rows.data_ptr(), dense, 0, s.csr.n_out, s.out.data_ptr(), dense)
    elif kind == "encrypt":
        gpu.encrypt_device(s.ctx, s.params, s.key, s.seed, s.n_rows, s.src.data_ptr(), s.geno.data_ptr(),
                           case["samples"], s.out.data_ptr() + 8, gpu.RECORD_OUT)
    elif kind == "decrypt":
        gpu.decrypt_device(s.ctx, s.key, s.rows.data_ptr(), dense, case["rows"], case["samples"], s.out.data_ptr())
    else:
        tickets = [s.server.submit(indiv, first, first + case["count"], h_in=h_in, h_out=h_out)
                   for indiv, first, h_in, h_out in s.requests]
        for t in tickets:
            s.server.wait(t)
        return [r[3] for r in s.requests]
    return s.out


def _neighbours(case):
    return case["neighbours"] or sum(UNEVEN) / len(UNEVEN)


def _tags_read(case):
    """Tags in at least one neighbourhood, when neighbourhoods hardly overlap."""
    return min(case["tags"], case["targets"] * _neighbours(case))


def work(case):
    """Inputs, weights and outputs once; an add or a multiply-add (two) per
    term, word and output.  Integer-polynomial weights count as the int16 a
    caller gives and their products as transforms of 5 N log2 N operations."""
    kind = case["kind"]
    row = 4 * 2 * N
    if kind in ("trlwe", "records", "range", "serve"):
        tags, targets, blocks = _tags_read(case), case["targets"], 1
        if kind in ("range", "serve"):
            tags = case["tags"] * case["count"] / case["targets"] + case["neighbours"]
            targets = case["count"]
        if kind == "serve":
            blocks = 1.5 * case["requests"]  # 1 .. 2,000 individuals in blocks of 1,024
        regions = _packing(case["samples"])[0] if kind != "serve" else 1
        terms = 3 * targets * 3 * case["neighbours"]
        return {"bytes": blocks * row * (3 * tags / regions + 3 * targets) + 8 * terms,
                "flops": blocks * 2 * terms * 2 * N}
    if kind == "lwe":
        words = case["indiv"] * (case["n"] + 1)
        terms = 3 * case["targets"] * 3 * _neighbours(case)
        return {"bytes": 4 * words * 3 * (_tags_read(case) + case["targets"]) + 8 * terms, "flops": 2 * terms * words}
    if kind in ("intpoly", "reweight"):
        terms = 3 * case["targets"] * 3 * case["neighbours"]
        transforms = 2 * 3 * (_tags_read(case) + case["targets"]) + (terms if kind == "reweight" else 0)
        return {"bytes": row * 3 * (_tags_read(case) + case["targets"]) + 2 * N * terms,
                "flops": terms * 2 * 2 * N + transforms * 5 * N * 10}
    if kind == "encrypt":
        rows = 3 * case["tags"] / _packing(case["samples"])[0]
        return {"bytes": row * rows + case["tags"] * case["samples"], "flops": rows * N * N / 2}
    return {"bytes": row * case["rows"] + 4 * case["rows"] * case["samples"],
            "flops": case["rows"] * case["samples"] * N / 2}


def _wrap32(x):
    return ((x + 2 ** 31) % 2 ** 32 - 2 ** 31).to(torch.int32)


def _exact_sums(csr, words_of, width, one):
    """sum of coef * row per output and its bias, int64, wrapped to 32 bits by the caller."""
    ptr = torch.from_numpy(csr.term_ptr.astype(np.int64)).cuda()
    feat = torch.from_numpy(csr.term_feat.astype(np.int64)).cuda()
    coef = torch.from_numpy(csr.term_coef.astype(np.int64)).cuda()
    n_out = csr.n_out
    step = max(1, (1 << 27) // width)
    for lo in range(0, n_out, step):
        hi = min(n_out, lo + step)
        acc = torch.zeros((hi - lo, width), dtype=torch.int64, device="cuda")
        bias = torch.zeros(hi - lo, dtype=torch.int64, device="cuda")
        longest = int((ptr[lo + 1:hi + 1] - ptr[lo:hi]).max())
        for t in range(longest):
            at = ptr[lo:hi] + t
            live = at < ptr[lo + 1:hi + 1]
            at = torch.where(live, at, torch.zeros_like(at))
            c = torch.where(live, coef[at], torch.zeros_like(at))
            f = feat[at]
            const = f == CONSTANT
            bias += torch.where(const, c * one, torch.zeros_like(c))
            c = torch.where(const, torch.zeros_like(c), c)
            f = torch.where(const, torch.zeros_like(f), f)
            acc += c[:, None] * words_of(f)
        yield lo, hi, acc, bias


def exact(case, seed):
    kind = case["kind"]
    if kind == "decrypt":
        s = prepare(case, seed)
        key = torch.from_numpy(s.key).cuda().to(torch.float64)
        # negacyclic Toeplitz matrix of the key: (a * key)[j] = sum_i a[i] T[i][j]
        d = (torch.arange(N, device="cuda")[None, :] - torch.arange(N, device="cuda")[:, None])
        toeplitz = torch.where(d >= 0, key[d % N], -key[d % N])[:, :case["samples"]].contiguous()
        out = torch.empty((case["rows"], case["samples"]), dtype=torch.float64, device="cuda")
        for lo in range(0, case["rows"], 16384):
            a = s.rows[lo:lo + 16384]
            product = (a[:, :N].to(torch.float64) @ toeplitz).to(torch.int64)  # below 2^41: exact
            phase = _wrap32(a[:, N:N + case["samples"]].to(torch.int64) - product)
            out[lo:lo + 16384] = phase.to(torch.float64) / 2.0 ** 32
        return out
    if kind == "trlwe":
        s = prepare(case, seed)
        j = torch.arange(N, device="cuda")

        def words_of(f):
            if s.regions == 1:
                return s.rows[f].to(torch.int64)
            at = j[None, :] + (f % s.regions)[:, None] * s.rs  # X^(-m) row, per polynomial
            sign = torch.where(at < N, 1, -1)
            rows = s.rows[f // s.regions].to(torch.int64)
            return torch.cat([rows[:, :N].gather(1, at % N) * sign, rows[:, N:].gather(1, at % N) * sign], 1)

        out = torch.empty_like(s.out)
        for lo, hi, acc, bias in _exact_sums(s.csr, words_of, 2 * N, gpu.ONE_IN_T32):
            acc[:, N:N + case["samples"]] += bias[:, None]
            acc[:, N + s.rs:] = 0
            out[lo:hi] = _wrap32(acc)
        return out
    if kind == "lwe":
        s = prepare(case, seed)
        words, n1 = case["indiv"] * (case["n"] + 1), case["n"] + 1
        out = torch.zeros_like(s.out)
        for lo, hi, acc, bias in _exact_sums(s.csr, lambda f: s.rows[f, :words].to(torch.int64), words,
                                             gpu.ONE_IN_T32):
            acc[:, n1 - 1::n1] += bias[:, None]
            out[lo:hi, :words] = _wrap32(acc)
        return out
    return None  # whole numbers of another generator, or of a schoolbook product that would take minutes
