"""
What the speed of this framework is measured on: single local operations of a sweep
(operator applies, environment steps, the QR and SVD of a site split), whole TDVP time
steps and a whole DMRG call, each through the public entry point a program calls, from
the README chain (bonds up to 28) to bonds of 1024.

Inputs are seeded. Local operations get device tensors: isometric site tensors, Hermitian
environments with an identity channel, the bulk tensor of the XXZ or Ising MPO. Whole
calls get a random MPS (bonds min(2^i, 2^(L-i), D)), as the tests and bench.py do.
exact() restates each operation in plain torch / NumPy complex128.
"""

import math

import numpy as np
import torch

import pytenet_gb300 as ptg

DEV = "cuda" if torch.cuda.is_available() else "cpu"
DT = 0.05j
J, DELTA, H = 1.0, 0.8, -0.1


# ------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call of an interactive user: one operator apply at bond 16, all latency
        dict(name="heff fp64 16", op="heff", prec="fp64", model="xxz", dl=16, dr=16),
        # default precision at the plain configuration's bond, one side ragged
        dict(name="heff fp64 250x256", op="heff", prec="fp64", model="xxz", dl=250, dr=256),
        # mixed precision at the headline bond
        dict(name="heff mixed 512", op="heff", prec="mixed", model="xxz", dl=512, dr=512),
        # an odd, rectangular environment step of the Ising batch's kind (left to right)
        dict(name="env left fp64 187x300", op="env_left", prec="fp64", model="ising", dl=187,
             dr=300),
        # environment step at the precision configuration's bond (right to left)
        dict(name="env right mixed 1024", op="env_right", prec="mixed", model="xxz", dl=1024,
             dr=1024),
        # QR of the bulk site tensor at bond 512: the orthonormalisation of every sweep step
        dict(name="qr 1024x512", op="qr", m=1024, n=512, sectors=1),
        # block QR of a U(1) state with odd sector sizes
        dict(name="qr u1 366x181", op="qr", m=366, n=181, sectors=5),
        # singular value decomposition of a two-site split, no symmetry
        dict(name="svd 128x96", op="svd", m=128, n=96),
        # the README run: ten sites, bonds up to 28, Lanczos depth 5, graph replay
        dict(name="tdvp fp64 L10 D28", op="tdvp", prec="fp64", sites=10, bond=28, depth=5,
             learned=False),
        # default precision on a chain with ragged bulk bonds, Lanczos depth 10
        dict(name="tdvp fp64 L20 D180", op="tdvp", prec="fp64", sites=20, bond=180, depth=10,
             learned=False),
        # the headline form: mixed precision, learned depth, bond 512
        dict(name="tdvp mixed L24 D512", op="tdvp", prec="mixed", sites=24, bond=512, depth=10,
             learned=True),
        # a whole DMRG call from host to host with conserved magnetisation
        dict(name="dmrg fp64 u1 L12 D24", op="dmrg", sites=12, bond=24, depth=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["heff", "heff", "bond", "env_left", "env_right", "qr", "qr", "svd", "tdvp",
                     "tdvp", "dmrg"])
    if op in ("heff", "bond", "env_left", "env_right"):
        prec = rng.choice(["fp64", "mixed"])
        dl = _log_int(rng, 8 if prec == "fp64" else 32, 1024)
        dr = min(1024, max(8, int(round(dl * rng.choice([0.5, 0.75, 1.0, 1.0, 1.3, 2.0])))))
        dr += rng.choice([0, 0, 1, -1, 3]) if dr < 1020 else 0
        return dict(op=op, prec=prec, model=rng.choice(["xxz", "ising"]), dl=dl, dr=dr)
    if op == "qr":
        n = _log_int(rng, 8, 768)
        m = max(4, int(round(n * rng.choice([0.5, 1.0, 2.0, 2.0, 2.0, 1.7]))) + rng.randint(-2, 2))
        return dict(op=op, m=m, n=n, sectors=rng.choice([1, 1, 3, 7]))
    if op == "svd":
        m = _log_int(rng, 6, 160)
        n = max(4, int(round(m * rng.uniform(0.5, 2.0))))
        return dict(op=op, m=m, n=min(n, 160))
    if op == "tdvp":
        prec = rng.choice(["fp64", "mixed"])
        bond = _log_int(rng, 8, 160 if prec == "fp64" else 300)
        return dict(op=op, prec=prec, sites=rng.randint(8, 20), bond=bond,
                    depth=rng.randint(4, 12), learned=prec == "mixed" and rng.random() < 0.5)
    return dict(op=op, sites=rng.randint(8, 12), bond=_log_int(rng, 16, 32),
                depth=rng.randint(5, 12))


# ------------------------------------------------------------------------ inputs
def _bulk_w(model):
    if model == "xxz":
        return torch.as_tensor(ptg.heisenberg_xxz_1d_mpo(8, J, DELTA, H).a[3], device=DEV,
                               dtype=torch.complex128).contiguous()
    return torch.as_tensor(ptg.ising_1d_mpo(8, J, 0.1, 1.1).a[3], device=DEV,
                           dtype=torch.complex128).contiguous()


def _gauss(gen, *shape):
    return torch.randn(*shape, dtype=torch.complex128, device=DEV, generator=gen)


def _isometry(gen, dl, d, dr):
    """Site tensor normalised as a whole, entries of a random state."""
    a = _gauss(gen, dl, d, dr)
    return (a / torch.linalg.vector_norm(a)).contiguous()


def _environment(gen, bond, chi, unit):
    """Hermitian operator blocks of order one, channel `unit` the identity."""
    e = _gauss(gen, bond, chi, bond) / math.sqrt(bond)
    e = 0.5 * (e + e.conj().permute(2, 1, 0))
    e[:, unit, :] = torch.eye(bond, dtype=torch.complex128, device=DEV)
    return e.contiguous()


def _local(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    w = _bulk_w(case["model"])
    d, chi = w.shape[1], w.shape[0]
    dl, dr = case["dl"], case["dr"]
    s = dict(w=w, a=_isometry(gen, dl, d, dr))
    if case["op"] in ("heff", "bond", "env_left"):
        s["l"] = _environment(gen, dl, chi, 0)
    if case["op"] in ("heff", "bond", "env_right"):
        s["r"] = _environment(gen, dr, chi, chi - 1)
    if case["op"] == "bond":
        s["c"] = s["a"][:, 0, :].contiguous()
    return s


def _sector_numbers(count, sectors):
    """Quantum numbers of a bond: binomially weighted sectors, shuffled as sweeps leave them."""
    if sectors == 1:
        return np.zeros(count, dtype=int)
    wt = np.array([math.comb(sectors - 1, k) for k in range(sectors)], float)
    edges = np.round(np.cumsum(wt) / wt.sum() * count).astype(int)
    q = 2 * np.searchsorted(edges, np.arange(count), side="right") - (sectors - 1)
    return np.random.default_rng(count).permutation(q)


def _matrix(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    m, n = case["m"], case["n"]
    a = _gauss(gen, m, n) / math.sqrt(n)
    q0, q1 = (_sector_numbers(x, case.get("sectors", 1)) for x in (m, n))
    if case.get("sectors", 1) > 1:
        a *= torch.as_tensor(q0[:, None] == q1[None, :], device=DEV)
    return a.contiguous(), q0, q1


def _hamiltonian(case):
    h = ptg.heisenberg_xxz_1d_mpo(case["sites"], J, DELTA, H)
    if case["op"] == "tdvp":
        h.zero_qnumbers()
    return h


def _state(case, seed, h):
    rng = np.random.default_rng(seed)
    n = case["sites"]
    if case["op"] == "dmrg":
        return ptg.MPS.construct_random(n, h.qsite, n % 2, case["bond"], rng=rng)
    b = [min(2 ** min(i, n - i), case["bond"]) for i in range(n + 1)]
    psi = ptg.MPS(h.qsite, [x * [0] for x in b], fill="random", rng=rng)
    for i, a in enumerate(psi.a):
        # isometries from both ends: a state without needlessly small Schmidt values
        if i < n // 2:
            psi.a[i] = np.linalg.qr(a.reshape(-1, a.shape[2]))[0].reshape(a.shape)
        else:
            psi.a[i] = np.linalg.qr(a.reshape(a.shape[0], -1).T)[0].T.reshape(a.shape)
    return psi


def prepare(case, seed):
    op = case["op"]
    if op in ("heff", "bond", "env_left", "env_right"):
        return dict(case, **_local(case, seed))
    if op in ("qr", "svd"):
        a, q0, q1 = _matrix(case, seed)
        return dict(case, a=a, q0=q0, q1=q1)
    h = _hamiltonian(case)
    psi = _state(case, seed, h)
    if op == "dmrg":
        return dict(case, h=h, psi=psi)
    model = None
    if case["learned"]:
        from pytenet_gb300.learned import DepthModel
        model = DepthModel.load()
    return dict(case, evolution=ptg.TDVPRun(h, psi, numiter_lanczos=case["depth"],
                                            precision=case["prec"], graph=True,
                                            depth_model=model))


# --------------------------------------------------------------------------- run
def _fixed_gauge(u, vh):
    """Singular vectors are defined up to a phase: the largest entry of every column of u
    becomes real and positive."""
    top = torch.gather(u, 0, u.abs().argmax(dim=0, keepdim=True))[0]
    ph = top.conj() / top.abs()
    return u * ph, vh * ph.conj()[:, None]


def _fixed_phase(v):
    top = v[np.argmax(np.abs(v))]
    return v * (top.conj() / abs(top))


def run(s):
    op = s["op"]
    if op == "heff":
        return ptg.apply_local_hamiltonian(s["a"], s["w"], s["l"], s["r"], precision=s["prec"])
    if op == "bond":
        return ptg.apply_local_bond_contraction(s["c"], s["l"], s["r"], precision=s["prec"])
    if op == "env_left":
        return ptg.contraction_operator_step_left(s["a"], s["a"], s["w"], s["l"],
                                                  precision=s["prec"])
    if op == "env_right":
        return ptg.contraction_operator_step_right(s["a"], s["a"], s["w"], s["r"],
                                                   precision=s["prec"])
    if op == "qr":
        return ptg.block_sparse_qr(s["a"], s["q0"], s["q1"])
    if op == "svd":
        u, sv, vh, q = ptg.block_sparse_svd(s["a"], s["q0"], s["q1"])
        u, vh = _fixed_gauge(u, vh)
        return u, sv, vh, q
    if op == "tdvp":
        # one symmetric time step of the resident state
        s["evolution"].step(DT)
        return s["evolution"].tensors()
    # one DMRG sweep of a fresh copy of the container (the call replaces its tensors)
    psi = ptg.MPS(s["psi"].qsite, s["psi"].qbonds, fill="postpone")
    psi.a = list(s["psi"].a)
    en = ptg.dmrg_singlesite(s["h"], psi, 1, numiter_lanczos=s["depth"])
    # the state as a vector: its tensors alone leave the gauge on the bonds open
    v = psi.to_vector()
    return en, np.concatenate(psi.qbonds), _fixed_phase(v)


# -------------------------------------------------------------------------- work
def _heff_flops(dl, d, dr, chi):
    return 8 * dl * d * chi * dr * dr + 8 * dl * dl * chi * d * dr


def _bond_flops(dl, dr, chi):
    return 8 * dl * chi * dr * dr + 8 * dl * dl * chi * dr


def _qr_flops(m, n):
    k = min(m, n)
    return 16 * (m * n * k - (m + n) * k * k / 2 + k ** 3 / 3)


def work(case):
    op = case["op"]
    if op in ("heff", "bond", "env_left", "env_right"):
        dl, dr, d = case["dl"], case["dr"], 2
        chi = 5 if case["model"] == "xxz" else 3
        le, re, a = dl * dl * chi, dr * dr * chi, dl * d * dr
        if op == "heff":
            return dict(bytes=16 * (2 * a + le + re), flops=_heff_flops(dl, d, dr, chi))
        if op == "bond":
            return dict(bytes=16 * (2 * dl * dr + le + re), flops=_bond_flops(dl, dr, chi))
        if op == "env_left":
            fl = 8 * dl * chi * dl * d * dr + 8 * dr * dl * d * chi * dr
        else:
            fl = 8 * dl * d * dr * chi * dr + 8 * dl * chi * d * dr * dl
        return dict(bytes=16 * (a + le + re), flops=fl)
    if op in ("qr", "svd"):
        m, n = case["m"], case["n"]
        k = min(m, n)
        if op == "svd":
            return dict(bytes=16 * (m * n + m * k + k * n), flops=16 * m * n * k + 32 * k ** 3)
        q0, q1 = (_sector_numbers(x, case["sectors"]) for x in (m, n))
        blocks = [(int((q0 == q).sum()), int((q1 == q).sum())) for q in np.intersect1d(q0, q1)]
        return dict(bytes=16 * (m * n + (m + n) * sum(min(b) for b in blocks)),
                    flops=sum(_qr_flops(*b) for b in blocks))
    n, chi, d = case["sites"], 5, 2
    b = [min(2 ** min(i, n - i), case["bond"]) for i in range(n + 1)]
    depth = case["depth"]
    fl = by = 0
    for i in range(n):
        dl, dr = b[i], b[i + 1]
        applies = 2 * depth * _heff_flops(dl, d, dr, chi)
        if op == "tdvp":
            applies += depth * (_bond_flops(dl, dl, chi) + _bond_flops(dr, dr, chi))
        fl += applies + _heff_flops(dl, d, dr, chi) * 2 + _qr_flops(dl * d, dr) + _qr_flops(
            dr * d, dl)
        by += 16 * (2 * dl * d * dr + dl * dl * chi + dr * dr * chi)
    return dict(bytes=2 * by, flops=fl)


# ------------------------------------------------------------------------- exact
def _x_heff(x, w, l, r):
    t = torch.tensordot(x, r, ([2], [0]))                # l0 t wr r2
    t = torch.tensordot(w, t, ([2, 3], [1, 2]))          # wl s l0 r2
    return torch.tensordot(l, t, ([0, 1], [2, 0]))       # l2 s r2


def _x_bond(c, l, r):
    return torch.tensordot(l, torch.tensordot(c, r, ([1], [0])), ([0, 1], [0, 1]))


def _x_env_left(a, w, l):
    t = torch.tensordot(l, a.conj(), ([2], [0]))         # l0 wl t rb
    t = torch.tensordot(w, t, ([0, 1], [1, 2]))          # s wr l0 rb
    return torch.tensordot(a, t, ([0, 1], [2, 0])).contiguous()   # ra wr rb


def _x_env_right(a, w, r):
    t = torch.tensordot(a, r, ([2], [0]))                # la s wr r2
    t = torch.tensordot(t, w, ([1, 2], [2, 3]))          # la r2 wl t
    return torch.tensordot(t, a.conj(), ([3, 1], [1, 2])).contiguous()   # la wl lb


def _x_qr(a, q0, q1):
    """Block QR with LAPACK factors, blocks in ascending order of their quantum number."""
    m, n = a.shape
    common = np.intersect1d(q0, q1)
    q, r, qi, k = [], [], [], 0
    for c in common:
        rows, cols = np.where(q0 == c)[0], np.where(q1 == c)[0]
        bq, br = np.linalg.qr(a[np.ix_(rows, cols)])
        fq = np.zeros((m, bq.shape[1]), complex)
        fr = np.zeros((bq.shape[1], n), complex)
        fq[rows], fr[:, cols] = bq, br
        q.append(fq)
        r.append(fr)
        qi.append(np.full(bq.shape[1], c))
    if len(common) == 0:
        e = np.zeros((m, 1), complex)
        e[0] = 1
        return e, np.zeros((1, n), complex), np.asarray(q0[:1])
    return np.concatenate(q, 1), np.concatenate(r, 0), np.concatenate(qi)


def _x_lanczos(apply, v, depth):
    shape, n = v.shape, v.numel()
    nrm = float(torch.linalg.vector_norm(v))
    vs, alpha, beta = [v.reshape(-1) / nrm], [], []
    for j in range(depth):
        y = apply(vs[j].reshape(shape)).reshape(-1)
        alpha.append(float(torch.vdot(y, vs[j]).real))
        if j == depth - 1:
            break
        y = y - alpha[j] * vs[j] - (beta[j - 1] * vs[j - 1] if j else 0)
        b = float(torch.linalg.vector_norm(y))
        if b < 100 * n * np.finfo(float).eps:
            break
        beta.append(b)
        vs.append(y / b)
    t = np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1)
    return nrm, t, torch.stack(vs, 1)


def _x_expm(apply, v, dt, depth):
    nrm, t, vs = _x_lanczos(apply, v, depth)
    w, u = np.linalg.eigh(t)
    c = nrm * (u @ (np.exp(-dt * w) * u[0]))
    return (vs @ torch.as_tensor(c, device=DEV)).reshape(v.shape)


def _x_lowest(apply, v, depth):
    _, t, vs = _x_lanczos(apply, v, depth)
    w, u = np.linalg.eigh(t)
    return w[0], (vs @ torch.as_tensor(u[:, 0].astype(complex), device=DEV)).reshape(v.shape)


class _Chain:
    """Reference sweep: right-normalised MPS, environments, local steps."""

    def __init__(self, h, psi, depth):
        def up(x):
            return torch.as_tensor(np.asarray(x, dtype=complex), device=DEV)
        self.a = [up(x) for x in psi.a]
        self.w = [up(x) for x in h.a]
        self.qs = np.asarray(psi.qsite)
        self.qb = [np.asarray(q) for q in psi.qbonds]
        self.depth, self.n = depth, len(psi.a)
        for i in reversed(range(1, self.n)):
            self.a[i - 1] = torch.tensordot(self.a[i - 1], self.right(i), ([2], [0]))
        if float(self.right(0)[0, 0].real) < 0:
            self.a[0] = -self.a[0]
        one = torch.ones((1, 1, 1), dtype=torch.complex128, device=DEV)
        self.l, self.r = [one] * self.n, [one] * self.n
        for i in reversed(range(1, self.n)):
            self.env_right(i)

    def left(self, i):
        a = self.a[i]
        q0 = np.add.outer(self.qb[i], self.qs).reshape(-1)
        q, r, self.qb[i + 1] = _x_qr(a.reshape(-1, a.shape[2]).cpu().numpy(), q0, self.qb[i + 1])
        self.a[i] = torch.as_tensor(q, device=DEV).reshape(a.shape[0], a.shape[1], -1)
        return torch.as_tensor(r, device=DEV)

    def right(self, i):
        a = self.a[i].permute(2, 1, 0)
        q0 = np.add.outer(-self.qb[i + 1], self.qs).reshape(-1)
        q, r, qi = _x_qr(a.reshape(-1, a.shape[2]).cpu().numpy(), q0, -self.qb[i])
        self.qb[i] = -qi
        self.a[i] = torch.as_tensor(q, device=DEV).reshape(a.shape[0], a.shape[1],
                                                           -1).permute(2, 1, 0).contiguous()
        return torch.as_tensor(r, device=DEV).T.contiguous()

    def env_left(self, i):
        self.l[i + 1] = _x_env_left(self.a[i], self.w[i], self.l[i])

    def env_right(self, i):
        self.r[i - 1] = _x_env_right(self.a[i], self.w[i], self.r[i])

    def heff(self, i):
        return lambda x: _x_heff(x, self.w[i], self.l[i], self.r[i])

    def tdvp_step(self, dt):
        n = self.n
        for i in range(n - 1):
            self.a[i] = _x_expm(self.heff(i), self.a[i], 0.5 * dt, self.depth)
            c = self.left(i)
            self.env_left(i)
            c = _x_expm(lambda x: _x_bond(x, self.l[i + 1], self.r[i]), c, -0.5 * dt, self.depth)
            self.a[i + 1] = torch.tensordot(c, self.a[i + 1], ([1], [0]))
        self.a[n - 1] = _x_expm(self.heff(n - 1), self.a[n - 1], dt, self.depth)
        for i in reversed(range(1, n)):
            c = self.right(i)
            self.env_right(i)
            c = _x_expm(lambda x: _x_bond(x, self.l[i], self.r[i - 1]), c, -0.5 * dt, self.depth)
            self.a[i - 1] = torch.tensordot(self.a[i - 1], c, ([2], [0]))
            self.a[i - 1] = _x_expm(self.heff(i - 1), self.a[i - 1], 0.5 * dt, self.depth)

    def dmrg_sweep(self):
        for i in range(self.n - 1):
            _, self.a[i] = _x_lowest(self.heff(i), self.a[i], self.depth)
            self.a[i + 1] = torch.tensordot(self.left(i), self.a[i + 1], ([1], [0]))
            self.env_left(i)
        for i in reversed(range(1, self.n)):
            en, self.a[i] = _x_lowest(self.heff(i), self.a[i], self.depth)
            self.a[i - 1] = torch.tensordot(self.a[i - 1], self.right(i), ([2], [0]))
            self.env_right(i)
        self.right(0)
        return en


def exact(case, seed):
    op = case["op"]
    if op in ("heff", "bond", "env_left", "env_right"):
        s = _local(case, seed)
        if op == "heff":
            return _x_heff(s["a"], s["w"], s["l"], s["r"])
        if op == "bond":
            return _x_bond(s["c"], s["l"], s["r"])
        if op == "env_left":
            return _x_env_left(s["a"], s["w"], s["l"])
        return _x_env_right(s["a"], s["w"], s["r"])
    if op in ("qr", "svd"):
        a, q0, q1 = _matrix(case, seed)
        if op == "qr":
            q, r, qi = _x_qr(a.cpu().numpy(), q0, q1)
            return torch.as_tensor(q), torch.as_tensor(r), qi
        u, sv, vh = np.linalg.svd(a.cpu().numpy(), full_matrices=False)
        u, vh = _fixed_gauge(torch.as_tensor(u), torch.as_tensor(vh))
        return u, sv, vh, np.zeros(len(sv), dtype=int)
    h = _hamiltonian(case)
    c = _Chain(h, _state(case, seed, h), case["depth"])
    if op == "tdvp":
        c.tdvp_step(DT)
        return c.a
    en = c.dmrg_sweep()
    v = c.a[0]
    for x in c.a[1:]:
        v = torch.tensordot(v, x, ([-1], [0]))
    return np.array([en]), np.concatenate(c.qb), _fixed_phase(v.reshape(-1).cpu().numpy())
