"""Scratch where the device has no memory for what the residue products ask for: the DMMA
kernels run on their smaller workspace, as everything did before there were residues. The
allocator's refusal is simulated by size."""

import warnings

import numpy as np
import pytest
import torch


def short_of_memory(monkeypatch, limit, device=None):
    """torch.empty refuses byte buffers above `limit`; returns the sizes that were asked for."""
    real, asked = torch.empty, []

    def empty(*args, **kw):
        if kw.get("dtype") is torch.uint8:
            asked.append(args[0])
            if args[0] > limit:
                raise torch.cuda.OutOfMemoryError("simulated")
            kw.pop("device", None) if device == "cpu" else None
        return real(*args, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    return asked


def test_workspace_takes_what_there_is(monkeypatch):
    from pytenet_gb300 import _lib, device
    monkeypatch.setattr(device, "device", lambda: None)
    asked = short_of_memory(monkeypatch, 5000, "cpu")
    w = device.Workspace()
    assert w.get(1000).numel() == 1000
    with pytest.raises(torch.cuda.OutOfMemoryError):
        w.get(6000)
    buf, n = w.room(8000, lambda: 2000)      # refused, smaller than the least: replaced
    assert (buf.numel(), n) == (2000, 2000)
    asked.clear()
    assert w.room(9000, lambda: 1500)[1] == 2000 and asked == []   # not asked for again
    assert w.room(7000, lambda: 1500)[1] == 2000 and asked == [7000]
    assert w.room(4000, lambda: 1500)[1] == 4000                   # there is memory for that
    assert w.room(0, lambda: 0)[1] == 256
    with pytest.raises(torch.cuda.OutOfMemoryError):
        w.room(9000, lambda: 6000)
    w = device.Workspace(remember=False)
    for _ in range(2):
        asked.clear()
        assert w.room(9000, lambda: 2000)[1] == 2000 and asked[0] == 9000   # asked every time
    size = {_lib.PREC_FP64: 8000, _lib.PREC_SPLIT_BF16: 7000, _lib.PREC_FP64_DMMA: 3000}
    for prec, runs in ((_lib.PREC_FP64, _lib.PREC_FP64), (_lib.PREC_SPLIT_BF16, _lib.PREC_FP64),
                       (_lib.PREC_FP64_DMMA, _lib.PREC_FP64_DMMA)):
        with warnings.catch_warnings(record=True) as seen:
            warnings.simplefilter("always")
            buf, n, p = device.Workspace().for_precision(size.get, prec)
        assert (n, p) == (3000, runs) and len(seen) == (prec == _lib.PREC_SPLIT_BF16)


def test_least_workspaces_are_the_two_intermediates():
    from pytenet_gb300 import _lib
    L = _lib.load()
    al = lambda b: (b + 255) // 256 * 256
    for dl, d, dr, cl, cr in ((16, 2, 16, 5, 5), (250, 2, 256, 5, 3), (4096, 2, 4096, 5, 5)):
        t = 2 * al(dl * d * dr * max(cl, cr) * 16)
        dims = (dl, d, dr, cl, cr, _lib.PREC_FP64_DMMA)
        assert L.ptn_heff_workspace_bytes(*dims) == L.ptn_env_workspace_bytes(*dims) == t
        assert L.ptn_site_step_workspace_bytes(*dims) == t
        t = 2 * al(dl * dr * cl * 16)
        assert L.ptn_bond_workspace_bytes(dl, dr, cl, _lib.PREC_FP64_DMMA) == t
        assert L.ptn_bond_step_workspace_bytes(dl, dr, cl, _lib.PREC_FP64_DMMA) == t
        assert L.ptn_qr_least_workspace_bytes(dl * d, dr) <= L.ptn_qr_workspace_bytes(dl * d, dr)


def operands(dl, d, dr, chi):
    gen = torch.Generator(device="cuda").manual_seed(dl)
    c = lambda *s: torch.randn(*s, dtype=torch.complex128, device="cuda", generator=gen)
    return c(dl, d, dr), c(chi, d, d, chi), c(dl, chi, dl), c(dr, chi, dr)


def rel(x, y):
    return float(torch.linalg.vector_norm(x - y) / torch.linalg.vector_norm(y))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_contractions_short_of_memory(monkeypatch, precision):
    import pytenet_gb300 as ptg
    from pytenet_gb300 import _lib, chain_ops
    from pytenet_gb300.device import Workspace
    dl, d, dr, chi = 120, 2, 130, 4
    a, w, l, r = operands(dl, d, dr, chi)
    calls = (lambda p: ptg.apply_local_hamiltonian(a, w, l, r, precision=p),
             lambda p: ptg.apply_local_bond_contraction(a[:, 0].contiguous(), l, r, precision=p),
             lambda p: ptg.contraction_operator_step_left(a, a, w, l, precision=p),
             lambda p: ptg.contraction_operator_step_right(a, a, w, r, precision=p))
    limit = _lib.load().ptn_heff_workspace_bytes(dl, d, dr, chi, chi, _lib.PREC_FP64_DMMA)
    plain = []
    for f in calls:   # the DMMA kernels by name: with room for nothing else, and with all the room
        monkeypatch.setattr(chain_ops, "_WS", Workspace())
        x = f("fp64-dmma")
        monkeypatch.setattr(chain_ops, "_WS", Workspace())
        chain_ops._WS.get(1 << 28)
        assert torch.equal(f("fp64-dmma"), x)
        y = f("fp64")
        assert not torch.equal(x, y) and rel(x, y) < 1e-13
        plain.append(x)
    with monkeypatch.context() as m:
        short_of_memory(m, limit)
        for f, x in zip(calls, plain):
            m.setattr(chain_ops, "_WS", Workspace())
            if precision == "mixed":
                with pytest.warns(RuntimeWarning, match="no device memory"):
                    y = f(precision)
            else:
                y = f(precision)
            assert rel(y, x) < 1e-13


@pytest.mark.gpu
def test_runs_short_of_memory(monkeypatch):
    """A whole time step of every form on the DMMA kernels' scratch."""
    import pytenet_gb300 as ptg
    from pytenet_gb300 import _lib
    rng = np.random.default_rng(4)
    n, cap = 16, 128
    h = ptg.heisenberg_xxz_1d_mpo(n, 1.0, 0.8, -0.1)
    h.zero_qnumbers()
    psi = ptg.MPS(h.qsite, [min(2 ** min(i, n - i), cap) * [0] for i in range(n + 1)], fill="random",
                  rng=rng)

    def step(precision):
        p = ptg.MPS(psi.qsite, psi.qbonds, fill="postpone")
        p.a = [x.copy() for x in psi.a]
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            ptg.tdvp_singlesite(h, p, 0.05j, 1, numiter_lanczos=4, precision=precision)
        return p

    ref = step("fp64")
    limit = _lib.load().ptn_env_workspace_bytes(cap, 2, cap, 5, 5, _lib.PREC_FP64_DMMA)
    with monkeypatch.context() as m:
        asked = short_of_memory(m, limit)
        got = [step(p) for p in ("fp64", "mixed", "fp64-dmma")]
        assert max(asked) > limit
    for p in got:
        for x, y in zip(p.a, ref.a):
            assert np.linalg.norm(x - y) < 1e-10 * np.linalg.norm(y)
