"""Corners of the dispatch rules: block QRs inside a captured graph, one-panel QRs of wide
matrices, workspaces smaller than the queries ask for, infinities and NaNs through whole
contractions."""

import warnings

import numpy as np
import pytest

from test_gpu_blocksparse import u1_state

pytestmark = pytest.mark.gpu


def crandn(rng, *s):
    return rng.standard_normal(s) + 1j * rng.standard_normal(s)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_u1_steps_from_a_graph(precision):
    """The wide blocks of a U(1) state run on forked streams, narrow ones in one launch: captured
    and replayed, the steps give the same bits as run one by one."""
    import pytenet_gb300 as ptg
    rng = np.random.default_rng(3)
    n, cap = 24, 256
    h = ptg.heisenberg_xxz_1d_mpo(n, 1.0, 0.8, -0.1)
    psi = u1_state(ptg, h, n, cap, rng)
    psi.orthonormalize(mode="left")
    out = []
    for graph in (False, True):
        p = ptg.MPS(psi.qsite, psi.qbonds, fill="postpone")
        p.a = [x.copy() for x in psi.a]
        run = ptg.TDVPRun(h, p, numiter_lanczos=5, precision=precision, graph=graph)
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            for _ in range(5):
                run.step(0.02j)
        assert (run.graph is not None) == graph
        out.append(run.download())
    # sectors too wide for the one-launch QR, several at a bond, beside narrow ones
    sizes = [np.unique(q, return_counts=True)[1] for q in out[0].qbonds]
    assert max((x > 16).sum() for x in sizes) >= 4 and any(x.min() <= 16 for x in sizes)
    for x, y in zip(out[0].a, out[1].a):
        assert np.array_equal(x, y)


def check_qr(a, q, r):
    k = min(a.shape)
    tol = 16 * max(a.shape) * np.finfo(float).eps
    assert q.shape == (a.shape[0], k) and r.shape == (k, a.shape[1])
    assert np.abs(q.conj().T @ q - np.eye(k)).max() <= tol
    assert np.linalg.norm(q @ r - a) <= tol * np.linalg.norm(a)
    assert np.all(np.tril(r, -1) == 0)
    ref = np.linalg.qr(a)[1]   # LAPACK's reflectors have the same signs
    assert np.abs(r - ref).max() <= 64 * tol * np.abs(a).max()


@pytest.mark.parametrize("mn", [(1, 1), (1, 16), (2, 3), (7, 16), (15, 16), (16, 16), (9, 10), (1, 2)])
def test_one_panel_qr_of_wide_matrices(mn):
    import torch
    from pytenet_gb300 import _lib
    from pytenet_gb300.device import empty, ptr, stream_ptr, to_dev, to_host
    L = _lib.load()
    m, n = mn
    k = min(m, n)
    a = crandn(np.random.default_rng(m + 17 * n), m, n)
    da, q, r = to_dev(a.copy()), empty((m, k)), empty((k, n))
    wsb = L.ptn_qr_workspace_bytes(m, n)
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    _lib.check(L.ptn_qr(ptr(da), m, n, ptr(q), k, ptr(r), n, ptr(ws), wsb, stream_ptr()))
    check_qr(a, to_host(q), to_host(r))


def test_block_qr_of_wide_and_tall_blocks():
    """Blocks of one launch: wide, square, tall and one-row ones, beside two wide-column ones."""
    import pytenet_gb300 as ptg
    rows, cols = [3, 16, 1, 40, 7, 30], [16, 16, 9, 5, 8, 21]
    rng = np.random.default_rng(6)
    q0 = rng.permutation(np.repeat(np.arange(6), rows))
    q1 = rng.permutation(np.repeat(np.arange(6), cols))
    a = crandn(rng, len(q0), len(q1)) * (q0[:, None] == q1[None, :])
    q, r, qi = ptg.block_sparse_qr(a, q0, q1)
    for c in range(6):
        i, j, k = np.where(q0 == c)[0], np.where(q1 == c)[0], np.where(qi == c)[0]
        check_qr(a[np.ix_(i, j)], q[np.ix_(i, k)], r[np.ix_(k, j)])
    assert np.all(q[q0[:, None] != qi[None, :]] == 0) and np.all(r[qi[:, None] != q1[None, :]] == 0)


@pytest.mark.parametrize("mn", [(1024, 512), (700, 300)])
def test_qr_on_a_smaller_workspace(mn):
    """One byte less than the query asks for: Q by panel-wide updates."""
    import torch
    from pytenet_gb300 import _lib
    from pytenet_gb300.device import empty, ptr, stream_ptr, to_dev, to_host
    L = _lib.load()
    m, n = mn
    a = crandn(np.random.default_rng(m), m, n)
    wsb = L.ptn_qr_workspace_bytes(m, n)
    for less in (0, 1):
        da, q, r = to_dev(a.copy()), empty((m, n)), empty((n, n))
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        _lib.check(L.ptn_qr(ptr(da), m, n, ptr(q), n, ptr(r), n, ptr(ws), wsb - less, stream_ptr()))
        check_qr(a, to_host(q), to_host(r))


def contractions(Dl, d, Dr, cl, cr, a, w, l, r, c, r2, small):
    """Every contraction through the C entry points, on the workspace that the queries ask for, or
    (small) the two intermediates alone, which leaves the DMMA kernels."""
    import torch
    from pytenet_gb300 import _lib
    from pytenet_gb300.device import empty, ptr, stream_ptr, to_dev, to_host
    L = _lib.load()
    A, W, Lt, R, Cm, R2 = (to_dev(x) for x in (a, w, l, r, c, r2))
    st = stream_ptr()
    out = []

    def run(fn, wsb, shape, args, dims):
        x = empty(shape)
        chi = dims[2] if len(dims) == 3 else d * max(cl, cr)
        least = 2 * ((Dl * chi * Dr * 16 + 255) // 256 * 256)
        assert least < wsb
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        _lib.check(fn(*args, ptr(x), *dims, 0, ptr(ws), least if small else wsb, st))
        out.append(to_host(x))

    dims = (Dl, d, Dr, cl, cr)
    run(L.ptn_heff_apply, L.ptn_heff_workspace_bytes(*dims, 0), (Dl, d, Dr),
        (ptr(A), ptr(W), ptr(Lt), ptr(R)), dims)
    env = L.ptn_env_workspace_bytes(*dims, 0)
    run(L.ptn_env_step_left, env, (Dr, cr, Dr), (ptr(A), ptr(A), ptr(W), ptr(Lt)), dims)
    run(L.ptn_env_step_right, env, (Dl, cl, Dl), (ptr(A), ptr(A), ptr(W), ptr(R)), dims)
    run(L.ptn_bond_apply, L.ptn_bond_workspace_bytes(Dl, Dr, cl, 0), (Dl, Dr),
        (ptr(Cm), ptr(Lt), ptr(R2)), (Dl, Dr, cl))
    return out


def operands(rng, Dl, d, Dr, cl, cr):
    w = rng.standard_normal((cl, d, d, cr)) * (rng.uniform(size=(cl, d, d, cr)) < 0.4) + 0j
    return (crandn(rng, Dl, d, Dr), w, crandn(rng, Dl, cl, Dl), crandn(rng, Dr, cr, Dr),
            crandn(rng, Dl, Dr), crandn(rng, Dr, cl, Dr))


def test_contractions_on_a_smaller_workspace():
    """The DMMA kernels, the same result to rounding."""
    dims = (72, 2, 77, 4, 5)
    ops = operands(np.random.default_rng(8), *dims)
    for x, y in zip(contractions(*dims, *ops, False), contractions(*dims, *ops, True)):
        assert not np.array_equal(x, y)   # another kernel
        assert np.linalg.norm(x - y) < 1e-13 * np.linalg.norm(y)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["site", "left", "right", "mpo"])
def test_infinities_and_nans_through_contractions(bad, where):
    """Where the DMMA kernels give a number the residue products give it too, and nowhere else."""
    dims = (72, 2, 77, 4, 5)
    ops = list(operands(np.random.default_rng(9), *dims))
    at = {"site": 0, "mpo": 1, "left": 2, "right": 3}[where]
    i = tuple(s // 2 for s in ops[at].shape) if where != "mpo" else (2, 1, 1, 3)
    ops[at][i] = bad
    if where == "site":
        ops[4][3, 4] = 1j * bad
    if where == "right":
        ops[5][3, 1, 5] = bad
    for x, y in zip(contractions(*dims, *ops, False), contractions(*dims, *ops, True)):
        fx, fy = (np.isfinite(t.real) & np.isfinite(t.imag) for t in (x, y))
        assert np.array_equal(fx, fy)
        assert np.linalg.norm(x[fx] - y[fy]) <= 1e-13 * np.linalg.norm(y[fy])


def test_graph_keeps_the_plans_it_reads():
    """The kernels of a captured step read index maps that belong to QR plans: a plan cache that
    is emptied (as it is when it is full) must not free them, nor steps with another dt."""
    import gc
    import weakref
    import pytenet_gb300 as ptg
    from pytenet_gb300 import qnumber
    rng = np.random.default_rng(5)
    h = ptg.heisenberg_xxz_1d_mpo(10, 1.0, 0.8, -0.1)
    psi = u1_state(ptg, h, 10, 24, rng)
    psi.orthonormalize(mode="left")
    run = ptg.TDVPRun(h, psi, numiter_lanczos=4, graph=True)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        run.step(0.02j)
        assert run.graph is not None
        captured = list(run.chain.plans.values())
        maps = [m[0].data_ptr() for p in captured for e in p.dev_cache.values()
                if isinstance(e, list) for m in e]
        alive = [weakref.ref(p) for p in captured]
        del captured
        qnumber._PLANS.clear()
        run.use_graph = False
        run.step(0.01j)   # by new plans
        run.use_graph = True
        gc.collect()
        assert maps and all(r() is not None for r in alive)
        run.step(0.02j)   # the graph again
    assert all(np.isfinite(x).all() for x in run.download().a)
