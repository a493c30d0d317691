"""FP64 GEMM in the residue number system (csrc/rns.cu): against products formed in extended
precision and against the DMMA kernel, over the edges of its tiles, all operand forms, rows
that leave the FP64 range, and operands whose products all have one sign.

Bound: an operand row is rounded to 53 bits or more of its largest component, so one of K
terms is off by at most 4 * 2^-53 max|A row| max|B column| and a result by K times that,
plus its own rounding; the tolerance is twice that."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def zgemm(A, B, opa="N", opb="N", alpha=1.0, beta=0.0, C=None, rns=True):
    """op(A) op(B) through ptn_zgemm; rns=False: no workspace, so the DMMA kernel."""
    import torch
    from pytenet_gb300 import _lib
    from pytenet_gb300.device import to_dev, to_host, ptr, stream_ptr, zeros
    L = _lib.load()
    M, K = A.shape if opa in "NC" else A.shape[::-1]
    N = B.shape[1] if opb in "NC" else B.shape[0]
    dA, dB = to_dev(A), to_dev(B)
    dC = zeros((M, N)) if C is None else to_dev(C).clone()
    wsb = L.ptn_zgemm_workspace_bytes(M, N, K, 1)
    assert not rns or wsb > 0, "the shape should take the residue planes"
    ws = torch.empty(max(wsb, 256), dtype=torch.uint8, device="cuda")
    _lib.check(L.ptn_zgemm(opa.encode(), opb.encode(), M, N, K, _lib.cval(alpha), ptr(dA),
                           A.shape[1], 0, ptr(dB), B.shape[1], 0, _lib.cval(beta), ptr(dC), N, 0,
                           1, ptr(ws), wsb if rns else 0, stream_ptr()))
    out = to_host(dC)
    assert L.ptn_tc_error() == 0
    return out


def crandn(rng, *s):
    return rng.standard_normal(s) + 1j * rng.standard_normal(s)


def exact(A, B, rows, cols):
    """Rows x columns of A B in extended precision."""
    a, b = A[rows].astype(np.clongdouble), B[:, cols].astype(np.clongdouble)
    return np.stack([(a[i][:, None] * b).sum(axis=0) for i in range(len(rows))])


def errors(C, A, B, rng, count=24):
    rows = np.unique(np.r_[0, A.shape[0] - 1, rng.integers(0, A.shape[0], count)])
    cols = np.unique(np.r_[0, B.shape[1] - 1, rng.integers(0, B.shape[1], count)])
    ref = exact(A, B, rows, cols)
    scale = (np.abs(A[rows]).max(axis=1)[:, None] * np.abs(B[:, cols]).max(axis=0)[None, :])
    err = np.abs(C[np.ix_(rows, cols)].astype(np.clongdouble) - ref)
    tol = 2 * (4 * A.shape[1] * scale * 2.0 ** -53 + 2.0 ** -53 * np.abs(ref).astype(float))
    return err, tol


@pytest.mark.parametrize("mnk", [(128, 256, 128), (129, 257, 200), (500, 1280, 256), (130, 66, 700),
                                 (1024, 33, 321), (64, 128, 512), (33, 4100, 255), (300, 300, 257),
                                 (250, 512, 1280), (37, 70, 8192)])
def test_matches_extended_precision(mnk):
    M, N, K = mnk
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A, B = crandn(rng, M, K), crandn(rng, K, N)
    err, tol = errors(zgemm(A, B), A, B, rng)
    assert np.all(err <= tol), (err / tol).max()
    err0, _ = errors(zgemm(A, B, rns=False), A, B, np.random.default_rng(1))
    rms, rms0 = (float(np.sqrt((e.astype(float) ** 2).mean())) for e in (err, err0))
    print(f"{mnk}: rms error {rms:.2e}, DMMA kernel {rms0:.2e}")
    assert rms <= 1.1 * rms0


@pytest.mark.parametrize("opa", list("NTCH"))
@pytest.mark.parametrize("opb", list("NTCH"))
def test_operand_forms(opa, opb):
    rng = np.random.default_rng(5)
    M, N, K = 141, 203, 167
    f = {"N": lambda x: x, "T": lambda x: x.T, "C": np.conj, "H": lambda x: x.conj().T}
    A = crandn(rng, *((M, K) if opa in "NC" else (K, M)))
    B = crandn(rng, *((K, N) if opb in "NC" else (N, K)))
    C0 = crandn(rng, M, N)
    al, be = 0.7 - 0.2j, -1.3 + 0.4j
    got = zgemm(A, B, opa, opb, al, be, C0)
    ref = al * (f[opa](A) @ f[opb](B)) + be * C0
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("kind", ["constant", "positive", "alternating", "powers"])
def test_one_signed_sums_are_exact(kind):
    """Every product of one sign: the largest chunk sums there can be."""
    rng = np.random.default_rng(6)
    M, N, K = 140, 150, 1500
    if kind == "constant":
        A, B = np.full((M, K), 0.7123 + 0.4567j), np.full((K, N), 0.9876 - 0.1j)
    elif kind == "positive":
        A = rng.uniform(0.5, 1, (M, K)) + 1j * rng.uniform(0.5, 1, (M, K))
        B = rng.uniform(0.5, 1, (K, N)) + 0j
    elif kind == "alternating":
        s = (-1.0) ** np.arange(K)
        A, B = np.full((M, K), 0.999) * s + 0j, (np.full((K, N), 0.999) * s[:, None]) + 0j
    else:
        A = 2.0 ** rng.integers(-30, 1, (M, K)) + 0j
        B = 2.0 ** rng.integers(-30, 1, (K, N)) + 0j
    err, tol = errors(zgemm(A, B), A, B, rng)
    assert np.all(err <= tol), (err / tol).max()


def test_scales_zeros_and_range_ends():
    """Rows and columns of very different size, zero rows, and rows whose entries or results
    leave the normal range: as the DMMA kernel gives them."""
    rng = np.random.default_rng(7)
    M, N, K = 160, 170, 180
    A, B = crandn(rng, M, K), crandn(rng, K, N)
    A[3] = 0
    B[:, 5] = 0
    A[10] *= 1e-150
    B[:, 11] *= 1e140
    A[20] *= 1e-300
    B[:, 21] *= 1e-300
    A[30] *= 1e-320 / 1e-10 * 1e-10
    A[40] *= 1e300
    B[:, 41] *= 1e300
    got, ref = zgemm(A, B), zgemm(A, B, rns=False)
    assert np.all(got[3] == 0) and np.all(got[:, 5] == 0)
    with np.errstate(over="ignore", invalid="ignore"):
        scale = np.abs(A).max(axis=1)[:, None] * np.abs(B).max(axis=0)[None, :] * K
    fin = np.isfinite(ref.real) & np.isfinite(ref.imag)
    assert np.array_equal(fin, np.isfinite(got.real) & np.isfinite(got.imag))
    ok = fin & np.isfinite(scale)
    d = np.abs(np.where(ok, got, 0) - np.where(ok, ref, 0))
    assert np.all(d <= np.where(ok, 1e-14 * scale, 0) + 1e-321)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_infinities_and_nans(bad):
    """An infinity or NaN makes the same results infinite or NaN as in the DMMA kernel and
    leaves every other result alone."""
    rng = np.random.default_rng(8)
    M, N, K = 140, 130, 256
    A, B = crandn(rng, M, K), crandn(rng, K, N)
    A[0] = 0
    clean = zgemm(A, B)
    A[7, 3] = bad
    B[9, 15] = 1j * bad
    got, ref = zgemm(A, B), zgemm(A, B, rns=False)
    for part in (np.real, np.imag):
        g, r = part(got), part(ref)
        assert np.array_equal(np.isnan(g), np.isnan(r)) and np.array_equal(np.isinf(g), np.isinf(r))
    same = np.ones((M, N), bool)
    same[7] = False
    same[:, 15] = False
    assert np.array_equal(got[same], clean[same])


@pytest.mark.parametrize("dims", [(32, 2, 40, 3, 5), (33, 3, 37, 5, 4), (129, 2, 65, 5, 5), (40, 2, 1100, 3, 3)])
def test_mixed_contractions_in_residues(dims):
    """The mixed form of every contraction (40 bits and more per operand row) on odd bonds, a
    physical dimension of 3, unequal MPO bonds and rows longer than one CTA converts: within
    2^-38 of the row maxima per term, by the bound of the FP64 planes at 40 bits."""
    import pytenet_gb300 as ptg
    Dl, d, Dr, cl, cr = dims
    rng = np.random.default_rng(sum(dims))
    a, b = crandn(rng, Dl, d, Dr), crandn(rng, Dl, d, Dr)
    w = rng.standard_normal((cl, d, d, cr))
    w[np.abs(w) < 0.7] = 0.0
    l, r = crandn(rng, Dl, cl, Dl), crandn(rng, Dr, cr, Dr)
    for fn, args, tr in ((ptg.apply_local_hamiltonian, (a, w, l, r), None),
                         (ptg.contraction_operator_step_left, (a, b, w, l), None),
                         (ptg.contraction_operator_step_right, (a, b, w, r), None)):
        got, ref = fn(*args, precision="mixed"), fn(*args, precision="fp64")
        assert np.linalg.norm(got - ref) < 1e-11 * np.linalg.norm(ref), fn.__name__


# around the smallest products that take the residue planes (a million complex multiply-adds)
@pytest.mark.parametrize("mnk", [(32, 1000, 32), (33, 947, 33), (100, 100, 101), (1030, 32, 33),
                                 (47, 235, 94), (64, 250, 64)])
def test_smallest_products(mnk):
    M, N, K = mnk
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    A, B = crandn(rng, M, K), crandn(rng, K, N)
    err, tol = errors(zgemm(A, B), A, B, rng)
    assert np.all(err <= tol), (err / tol).max()


def spread(rng, n, width):
    """n factors between 1 / width and 1, both ends among them, in random order."""
    s = 10.0 ** -(rng.uniform(0, 1, n) * np.log10(width))
    s[rng.permutation(n)[:2]] = 1.0, 1.0 / width
    return s


# Operands that grow and decay against each other along the summed index: the products are of
# one size, so FP64 has them to rounding. Tolerance: the form's 1e-12 per contraction, in the
# norm without the scalings (rounding alone is below 1e-14 at these sizes).
GAUGES = [1e3, 1e6, 1e9, 1e12]


@pytest.mark.parametrize("width", GAUGES)
@pytest.mark.parametrize("ops", ["NN", "TN", "NT", "HC"])
@pytest.mark.parametrize("mnk", [(128, 130, 96), (40, 300, 700), (310, 36, 1100)])
def test_products_of_opposite_scalings(mnk, ops, width):
    """A D times D^-1 B, with rows of A and columns of B scaled too."""
    M, N, K = mnk
    rng = np.random.default_rng(M + K + int(np.log10(width)))
    s, x, y = spread(rng, K, width), spread(rng, M, width), spread(rng, N, 1e3)
    A = x[:, None] * crandn(rng, M, K) * s
    B = crandn(rng, K, N) / s[:, None] * y
    g = {"N": lambda z: z, "T": lambda z: z.T, "C": np.conj, "H": lambda z: z.conj().T}
    got = zgemm(np.ascontiguousarray(g[ops[0]](A)), np.ascontiguousarray(g[ops[1]](B)), *ops)
    rows, cols = rng.integers(0, M, 30), rng.integers(0, N, 30)
    ref = exact(A, B, rows, cols)
    free = x[rows][:, None] * y[cols][None, :]
    err = np.linalg.norm(((got[np.ix_(rows, cols)] - ref) / free).astype(complex))
    assert err < 1e-12 * np.linalg.norm((ref / free).astype(complex))


@pytest.mark.parametrize("channel", ["dense", "identity"])
@pytest.mark.parametrize("width", GAUGES)
def test_contractions_in_a_scaled_gauge(width, channel):
    """A site tensor in the gauge X a Y with the environments of that gauge: both products of
    every contraction sum over an index that the two operands scale against each other."""
    import pytenet_gb300 as ptg
    Dl, d, Dr, cl, cr = 72, 2, 76, 3, 4
    rng = np.random.default_rng(int(np.log10(width)))
    x, y = spread(rng, Dl, width), spread(rng, Dr, width)
    a, b = crandn(rng, Dl, d, Dr), crandn(rng, Dl, d, Dr)
    w = rng.standard_normal((cl, d, d, cr)) + 0j
    l, r, c = crandn(rng, Dl, cl, Dl), crandn(rng, Dr, cr, Dr), crandn(rng, Dl, Dr)
    r2 = crandn(rng, Dr, cl, Dr)
    if channel == "identity":
        l[:, 0], r[:, 0], r2[:, 0] = np.eye(Dl), np.eye(Dr), np.eye(Dr)
    # X a Y, X^-1 l X^-1, Y^-1 r Y^-1
    up = lambda t: x[:, None, None] * t * y[None, None, :]
    lx = l / (x[:, None, None] * x[None, None, :])
    ry, ry2 = (t / (y[:, None, None] * y[None, None, :]) for t in (r, r2))
    q = lambda t: t.astype(np.clongdouble)

    def close(got, ref, free):
        free = np.broadcast_to(free, got.shape)
        err = np.linalg.norm(((got - ref) * free).astype(complex))
        assert err < 1e-12 * np.linalg.norm((ref * free).astype(complex))

    A, B, W, L, R = (q(t) for t in (up(a), up(b), w, lx, ry))
    t1 = np.tensordot(A, R, ([2], [0]))                                  # l0 t wr r2
    t2 = np.tensordot(W, t1, ([2, 3], [1, 2]))                           # wl s l0 r2
    close(ptg.apply_local_hamiltonian(up(a), w, lx, ry), np.tensordot(L, t2, ([0, 1], [2, 0])),
          x[:, None, None] * y[None, None, :])
    cx = x[:, None] * c * y[None, :]
    ref = np.tensordot(L, np.tensordot(q(cx), q(ry2), ([1], [0])), ([0, 1], [0, 1]))
    close(ptg.apply_local_bond_contraction(cx, lx, ry2), ref, x[:, None] * y[None, :])
    t = np.tensordot(L, B.conj(), ([2], [0]))                            # l0 wl t rb
    t = np.tensordot(W, t, ([0, 1], [1, 2]))                             # s wr l0 rb
    ref = np.tensordot(A, t, ([0, 1], [2, 0]))                           # ra wr rb
    close(ptg.contraction_operator_step_left(up(a), up(b), w, lx), ref,
          1 / (y[:, None, None] * y[None, None, :]))
    t = np.tensordot(t1, W, ([1, 2], [2, 3]))                            # l0 r2 wl t
    ref = np.tensordot(t, B.conj(), ([3, 1], [1, 2]))                    # la wl lb
    close(ptg.contraction_operator_step_right(up(a), up(b), w, ry), ref,
          1 / (x[:, None, None] * x[None, None, :]))


def test_terms_that_meet_zeros_or_subnormals():
    """Terms without entries in one operand drop out whatever the other one holds there (but
    for infinities and NaNs), and subnormal entries count where their term is large."""
    rng = np.random.default_rng(11)
    M, N, K = 140, 150, 96
    A, B = crandn(rng, M, K), crandn(rng, K, N)
    B[5] = 0
    A[:, 5] *= 1e200
    A[:, 9] *= 2.0 ** -1050
    B[9] *= 2.0 ** 1000
    B[11] *= 2.0 ** -1060
    A[:, 11] *= 2.0 ** 1010
    got = zgemm(A, B)
    keep = np.arange(K) != 5
    err, tol = errors(got, np.delete(A, 5, 1) * 1.0, np.delete(B, 5, 0) * 1.0, rng)
    # rows and columns without the scalings, as bounds of the terms
    s = np.ones(K)
    s[9], s[11] = 2.0 ** 1000, 2.0 ** -1010
    As, Bs = (A * s)[:, keep], (B / s[:, None])[keep]
    bound = 32 * K * 2.0 ** -53 * np.abs(As).max() * np.abs(Bs).max()
    assert np.isfinite(got).all() and float(err.max()) < bound
    A[3, 5] = np.inf
    bad = zgemm(A, B)
    assert not np.isfinite(bad[3]).any() and np.isfinite(np.delete(bad, 3, 0)).all()


# Rows longer than a cluster converts (8192 terms): their exponents come from a pass of their
# own, 11 moduli leave 40 bits up to 16384 terms and 39 beyond, 13 moduli 49 and 48, and the
# FP64 form keeps to the DMMA kernels (fewer than 53 bits). Tolerance: rows of Gaussian entries
# reach 8, so an entry of order one is off by 2^(3 - bits) at most, in either operand, and the
# errors of the terms add up like the terms: twice 2^(3 - 39) and 2^(3 - 48).
@pytest.mark.parametrize("op,chi,tol", [("bond", 300, 2 * 2.0 ** -36), ("bond", 520, 2 * 2.0 ** -36),
                                        ("env", 3, 2 * 2.0 ** -45)])
def test_mixed_contractions_of_long_rows(op, chi, tol):
    import torch
    import pytenet_gb300 as ptg
    gen = torch.Generator(device="cuda").manual_seed(chi)
    c = lambda *s: torch.randn(*s, dtype=torch.complex128, device="cuda", generator=gen)
    if op == "bond":
        dl, dr = 33, 40
        args, fn = (c(dl, dr), c(dl, chi, dl), c(dr, chi, dr)), ptg.apply_local_bond_contraction
    else:
        dl, dr = 33, 4100
        w = torch.randn(chi, 2, 2, chi, dtype=torch.complex128, device="cuda", generator=gen)
        args = (c(dl, 2, dr), c(dl, 2, dr), w, c(dr, chi, dr))
        fn = ptg.contraction_operator_step_right
    got, ref = fn(*args, precision="mixed"), fn(*args, precision="fp64")
    err = float(torch.linalg.vector_norm(got - ref) / torch.linalg.vector_norm(ref))
    assert 0 < err < tol, err
