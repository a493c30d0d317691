"""A bounded wait that expires in a tensor-core kernel is reported: by NaN in everything the
residue products give while the error word stands, and by an exception wherever a result
reaches the host. The word is set from the host (ptn_device_error_inject); no wait runs out."""

import numpy as np
import pytest


class FakeLib:
    def __init__(self, code):
        self.code = code

    def ptn_device_error(self, stream):
        code, self.code = self.code, 0
        return code


@pytest.mark.parametrize("code,status", [(1, "PTN_TIMEOUT"), (3, "PTN_TIMEOUT"), (-1, "PTN_CUDA_ERROR")])
def test_host_reads_raise_on_the_error_word(monkeypatch, code, status):
    import torch
    from pytenet_gb300 import _lib, device

    class OnDevice:
        """As much of a CUDA tensor as a download uses."""
        is_cuda = True

        def __init__(self, x):
            self.x = x

        def detach(self):
            return self.x

        def reshape(self, *s):
            return OnDevice(self.x.reshape(*s))

        def __getitem__(self, i):
            return OnDevice(self.x[i])

    fake = FakeLib(code)
    monkeypatch.setattr(device, "lib", lambda: fake)
    monkeypatch.setattr(device, "stream_ptr", lambda: 0)
    t = OnDevice(torch.arange(3.0))
    for read in (device.to_host, device.scalar, lambda x: device.to_host_all([x, x])):
        fake.code = code
        with pytest.raises(_lib.PtnError) as e:
            read(t)
        assert e.value.status == getattr(_lib, status)
    # read once, the word is clear again; host tensors are not checked
    assert np.array_equal(device.to_host(t), np.arange(3.0))
    fake.code = code
    assert np.array_equal(device.to_host(torch.arange(3.0)), np.arange(3.0))


def inject(code):
    from pytenet_gb300 import _lib
    from pytenet_gb300.device import stream_ptr
    _lib.check(_lib.load().ptn_device_error_inject(code, stream_ptr()))


def operands(rng, dl, d, dr, chi):
    import torch
    c = lambda *s: torch.tensor(rng.standard_normal(s) + 1j * rng.standard_normal(s), device="cuda")
    return (c(dl, d, dr), torch.tensor(rng.standard_normal((chi, d, d, chi)) + 0j, device="cuda"),
            c(dl, chi, dl), c(dr, chi, dr))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_products_are_nan_while_the_word_stands(precision):
    import torch
    import pytenet_gb300 as ptg
    from pytenet_gb300 import _lib
    from pytenet_gb300.device import check_device, to_host
    a, w, l, r = operands(np.random.default_rng(1), 72, 2, 75, 4)
    calls = (lambda: ptg.apply_local_hamiltonian(a, w, l, r, precision=precision),
             lambda: ptg.apply_local_bond_contraction(a[:, 0].contiguous(), l, r, precision=precision),
             lambda: ptg.contraction_operator_step_left(a, a, w, l, precision=precision),
             lambda: ptg.contraction_operator_step_right(a, a, w, r, precision=precision))
    good = [to_host(f()) for f in calls]
    for f, ref in zip(calls, good):
        inject(2)
        bad = f()
        assert bool(torch.isnan(torch.view_as_real(bad)).all())
        with pytest.raises(_lib.PtnError) as e:
            to_host(bad)
        assert e.value.status == _lib.PTN_TIMEOUT
        assert np.array_equal(to_host(f()), ref)
    check_device()


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
def test_a_run_raises_instead_of_returning_tensors(graph):
    import pytenet_gb300 as ptg
    from pytenet_gb300 import _lib
    rng = np.random.default_rng(2)
    n, cap = 14, 64
    h = ptg.heisenberg_xxz_1d_mpo(n, 1.0, 0.8, -0.1)
    h.zero_qnumbers()
    psi = ptg.MPS(h.qsite, [min(2 ** min(i, n - i), cap) * [0] for i in range(n + 1)], fill="random",
                  rng=rng)
    run = ptg.TDVPRun(h, psi, numiter_lanczos=4, graph=graph)
    for _ in range(3):
        run.step(0.05j)
    before = [x.copy() for x in psi.a]
    inject(1)
    run.step(0.05j)
    with pytest.raises(_lib.PtnError):
        run.download()
    assert all(np.array_equal(x, y) for x, y in zip(before, psi.a))   # nothing was handed out


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["expm", "eigh", "python"])
def test_a_lanczos_run_that_timed_out_is_reported(mode):
    """The state of a Lanczos step whose grid barrier gave up, as that step leaves it."""
    import torch
    from pytenet_gb300 import _lib, krylov
    from pytenet_gb300.device import check_device, ptr, stream_ptr, to_dev, to_host
    rng = np.random.default_rng(3)
    r = krylov._Run(to_dev(rng.standard_normal(300) + 0j), 4)
    check_device()
    at = _lib.KrylovState.status.offset
    r.state[at:at + 4].view(torch.int32).fill_(_lib.PTN_TIMEOUT)
    L = _lib.load()
    if mode == "python":
        with pytest.raises(_lib.PtnError):
            r.read_state()
        return
    if mode == "expm":
        _lib.check(L.ptn_krylov_expm_coef(ptr(r.state), 0.0, -0.1, stream_ptr()))
    else:
        _lib.check(L.ptn_krylov_eigh_coef(ptr(r.state), stream_ptr()))
    with pytest.raises(_lib.PtnError) as e:
        to_host(r.V)
    assert e.value.status == _lib.PTN_TIMEOUT and "code 4" in str(e.value)
    check_device()
