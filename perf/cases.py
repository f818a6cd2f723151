"""Performance cases of the TD-SCHA linear-response engine.

Every case runs one call of a public entry point on a seeded rock-salt ensemble (the generator's
geometry, harmonic modes and symmetry group; anharmonic forces of the bond terms), over the range
that the tests and the benchmark cover: 2x2x2 to 4x4x4 supercells (45 to 381 modes, 384 to 3072
symmetry operations, or none), 200 to 10^4 configurations, 1 to 32 vectors per apply, FP64 and the
mixed precisions, the standard and the Wigner representation, L and its transpose, the averages'
gradient, the static operator, a whole chain and its continued fraction.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "python-sscha_b200"))
from tdscha_b200 import _native, rocksalt  # noqa: E402

T = 300.0
DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # G(w) of a finished chain on the 500-point grid of the 2x2x2 workload: the smallest call a
        # user makes, once per chain and smearing
        dict(name="green_100_500", kind="green", steps=100, points=500),
        # the plain FP64 workload: one chain on 2x2x2, N = 2000; every step is one apply of (q, p)
        dict(name="apply_l2_fp64_2", kind="apply", L=2, N=2000, nb=2, precision="fp64", wigner=False, group="full", reweighted=False),
        # the same chain driven on the device for 12 steps (start-up, captured steps, recurrence)
        dict(name="chain_l2_fp64_1x12", kind="chain", L=2, N=2000, chains=1, steps=12, precision="fp64", group="full", reweighted=False),
        # 16 chains (3 IR, 6 Raman, 7 random) batched over the small system
        dict(name="apply_l2_bf16x3_32", kind="apply", L=2, N=2000, nb=32, precision="bf16x3", wigner=False, group="full", reweighted=False),
        # an ensemble without symmetries (unsymmetrised run), odd sizes, reweighted configurations
        dict(name="apply_l2_nosym_tf32x3_3", kind="apply", L=2, N=1531, nb=3, precision="tf32x3", wigner=False, group="none", reweighted=True),
        # 16 chains batched over the middle system
        dict(name="apply_l3_bf16x3_32", kind="apply", L=3, N=5000, nb=32, precision="bf16x3", wigner=False, group="full", reweighted=False),
        # Wigner representation, ragged configuration count (a reweighted ensemble after rejection)
        dict(name="apply_l3_wigner_tf32x3_5", kind="apply", L=3, N=4999, nb=5, precision="tf32x3", wigner=True, group="full", reweighted=True),
        # free-energy Hessian: the static operator on the vectors of a batch of minimum-residual solves
        dict(name="static_l3_fp64_24", kind="static", L=3, N=1200, nb=24, precision="fp64", group="full", reweighted=False),
        # gradient of G(w): the averages' vector-Jacobian product of one chain's (q, p)
        dict(name="vjp_l3_bf16x3_2", kind="vjp", L=3, N=5000, nb=2, precision="bf16x3", group="full", reweighted=True),
        # one chain on the large system
        dict(name="apply_l4_bf16x3_2", kind="apply", L=4, N=10000, nb=2, precision="bf16x3", wigner=False, group="full", reweighted=False),
        # one FP64 step on the large system (the accuracy reference of the mixed chains)
        dict(name="apply_l4_fp64_2", kind="apply", L=4, N=10000, nb=2, precision="fp64", wigner=False, group="full", reweighted=False),
        # the benchmark workload: 8 chains on 4x4x4, N = 10^4
        dict(name="apply_l4_bf16x3_16", kind="apply", L=4, N=10000, nb=16, precision="bf16x3", wigner=False, group="full", reweighted=False),
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    cap = _cost(next(c for c in listed() if c["name"] == "apply_l4_bf16x3_16"))
    while True:
        kind = rng.choice(["apply", "apply", "apply", "apply", "apply", "static", "vjp", "chain", "green"])
        if kind == "green":
            return dict(kind=kind, steps=_log_int(rng, 20, 300), points=_log_int(rng, 100, 2000))
        L = rng.choice([2, 2, 3, 3, 4])
        N = _log_int(rng, 200, {2: 4000, 3: 6000, 4: 10000}[L])
        c = dict(kind=kind, L=L, N=N, precision=rng.choice(["fp64", "bf16x3", "bf16x3", "bf16x3", "tf32x3", "tf32"]),
                 group="none" if L == 2 and rng.random() < 0.2 else "full", reweighted=rng.random() < 0.5)
        if kind == "apply":
            c.update(nb=_log_int(rng, 1, 32), wigner=rng.random() < 0.3)
        elif kind == "static":
            c.update(nb=_log_int(rng, 4, 48))
        elif kind == "vjp":
            if L == 4:
                continue
            c.update(nb=_log_int(rng, 1, 4))
        else:
            if L == 4:
                continue
            c.update(chains=_log_int(rng, 1, 4), steps=rng.randint(4, 12))
        if _cost(c) <= cap:
            return c


def _cost(case):
    w = work(case)["flops"]
    return w * {"fp64": 10.0, "tf32x3": 2.0, "tf32": 0.7}.get(case.get("precision"), 1.0)


# ---- inputs -----------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _system(L, group):
    """Geometry, modes and symmetry tables (no seed enters them), and the map A with
    dr = X A (bond stretches of mode displacements), Y = -(k3/2 dr^2 + k4/6 dr^3) A^T."""
    full = group == "full"
    s = rocksalt.build_system(L, T=T, with_symmetries=full, symmetries_on_gpu=full)
    d = np.zeros((len(s.bonds), 3 * s.nat))
    for b, (i, j) in enumerate(s.bonds):
        d[b, 3 * i:3 * i + 3] = -s.bond_dirs[b]
        d[b, 3 * j:3 * j + 3] = s.bond_dirs[b]
    A = (s.pols.T / np.sqrt(s.masses)) @ d.T
    return s, A


def _bose(w):
    return 1.0 / (torch.exp(w * rocksalt.RY_TO_K / T) - 1.0)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, dtype=F64, device=DEV)


def _inputs(case, seed):
    """The seeded arrays of a case: ensemble (X, Y, rho) and vectors, float64 on the device."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    if case["kind"] == "green":
        # coefficients of a converged chain: a around the squared frequencies, b and c of one sign
        k = case["steps"]
        w2 = 1e-6
        a = w2 * (1.0 + 0.2 * _normal(g, k))
        b = w2 * (0.3 + 0.05 * torch.rand(k, generator=g, dtype=F64, device=DEV))
        c = w2 * (0.3 + 0.05 * torch.rand(k, generator=g, dtype=F64, device=DEV))
        omega = torch.linspace(0.0, 400.0 / rocksalt.RY_TO_CM, case["points"], dtype=F64, device=DEV)
        return dict(a=a, b=b, c=c, omega=omega)
    s, A = _system(case["L"], case["group"])
    w = torch.as_tensor(s.w, device=DEV)
    A = torch.as_tensor(A, device=DEV)
    n, N = s.n_modes, case["N"]
    X = _normal(g, N, n) * torch.sqrt((1.0 + 2.0 * _bose(w)) / (2.0 * w))
    dr = X @ A
    Y = -(s.k3 / 2 * dr ** 2 + s.k4 / 6 * dr ** 3) @ A.T
    # importance weights of an ensemble reused after a small change of the dynamical matrix
    rho = torch.exp(0.2 * _normal(g, N)) if case["reweighted"] else torch.ones(N, dtype=F64, device=DEV)
    d = dict(w=w, X=X, Y=Y, rho=rho)
    if case["kind"] == "vjp":
        def sym(nb):
            M = _normal(g, nb, n, n)
            return 0.5 * (M + M.transpose(1, 2))
        nb = case["nb"]
        d.update(R1=_normal(g, nb, n), Ys=sym(nb), fbar=_normal(g, nb, n), Dbar=sym(nb))
    elif case["kind"] == "chain":
        q = torch.zeros(case["chains"], n + n * (n + 1), dtype=F64, device=DEV)
        q[:, :n] = _normal(g, case["chains"], n)
        d["q"] = q / q.norm(dim=1, keepdim=True)
    else:
        P = n * (n + 1) // 2
        psi = _normal(g, case["nb"], n + (2 * P if case["kind"] == "apply" else P))
        d["psi"] = psi / psi.norm(dim=1, keepdim=True)
    return d


def _transpose(nb):
    """L on the first half of the vectors (q of every chain), its transpose on the rest (p)."""
    return [0] * ((nb + 1) // 2) + [1] * (nb // 2)


def prepare(case, seed):
    d = _inputs(case, seed)
    if case["kind"] == "green":
        d["gf"] = torch.empty(2 * case["points"], dtype=F64, device=DEV)
        return dict(case=case, **d)
    s, _ = _system(case["L"], case["group"])
    ens = _native.DeviceEnsemble(d["X"].cpu().numpy(), d["Y"].cpu().numpy(), s.w, d["rho"].cpu().numpy(), T, s.symmetries,
                                 s.deg_space, s.blocks_ids)
    st = dict(case=case, ens=ens)
    if case["kind"] == "vjp":
        st.update({k: d[k] for k in ("R1", "Ys", "fbar", "Dbar")})
        st.update(Ybar=torch.empty_like(d["Y"]), rhobar=torch.empty_like(d["rho"]))
    elif case["kind"] == "chain":
        nc = case["chains"]
        st["qp0"] = torch.stack([d["q"], d["q"], torch.zeros_like(d["q"]), torch.zeros_like(d["q"])])
        st["sc0"] = torch.tensor([[0.0, 0.0, 1.0, 0.0, 1.0, 0.0]] * nc, dtype=F64, device=DEV)
        st.update(qp=torch.empty_like(st["qp0"]), sc=torch.empty_like(st["sc0"]),
                  coef=torch.zeros(case["steps"], nc, 4, dtype=F64, device=DEV), opts=_native.ApplyOpts())
    else:
        st.update(psi=d["psi"], out=torch.empty_like(d["psi"]))
        if case["kind"] == "apply":
            st.update(opts=_native.ApplyOpts(use_wigner=int(case["wigner"])), transpose=_transpose(case["nb"]))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "apply":
        st["ens"].apply_full_L(st["psi"], st["out"], st["transpose"], st["opts"], precision=case["precision"])
        return st["out"]
    if kind == "static":
        _native.apply_static_L(st["ens"], st["psi"], st["out"], precision=case["precision"])
        return st["out"]
    if kind == "vjp":
        st["ens"].perturb_average_vjp(st["R1"], st["Ys"], st["fbar"], st["Dbar"], st["Ybar"], st["rhobar"],
                                      precision=case["precision"])
        return st["Ybar"], st["rhobar"]
    if kind == "chain":
        st["qp"].copy_(st["qp0"])
        st["sc"].copy_(st["sc0"])
        _native.lanczos_run([(st["ens"], st["qp"], st["sc"], st["coef"], st["opts"], case["precision"])], case["steps"])
        return st["coef"], st["qp"], st["sc"]
    _native.continued_fraction(st["a"], st["b"], st["c"], st["omega"], st["gf"], False, 1, 5.0 / rocksalt.RY_TO_CM, False,
                               False, 0.0, 1.0)
    return st["gf"]


def work(case):
    """Bytes: the ensemble and the vectors, each read once, and the outputs.  Flops: the two big
    contractions (configurations x packed mode pairs) over the 48 rotations and the characters of the
    L^3 translations (a complex character counts twice), a product counted once in every precision."""
    if case["kind"] == "green":
        return dict(bytes=8.0 * (3 * case["steps"] + 3 * case["points"]), flops=30.0 * case["steps"] * case["points"])
    L, N = case["L"], case["N"]
    n = 6 * L ** 3 - 3
    P = n * (n + 1) // 2
    rows = 1.0
    if case["group"] == "full":
        rows = 48 * (2.0 - (8 if L % 2 == 0 else 1) / L ** 3)
    ens = 8.0 * (2 * N * n + N)
    pair = 2.0 * 2 * N * rows * P   # one contraction of one vector
    if case["kind"] == "vjp":
        nb = case["nb"]
        return dict(bytes=ens + 16.0 * nb * (n + n * n) + 8.0 * (N * n + N), flops=3 * nb * pair)
    if case["kind"] == "chain":
        nb = 2 * case["chains"]
        return dict(bytes=case["steps"] * (ens + 32.0 * nb * (n + 2 * P)), flops=case["steps"] * nb * 2 * pair)
    vec = 16.0 * case["nb"] * (n + (2 * P if case["kind"] == "apply" else P))
    return dict(bytes=ens + vec, flops=case["nb"] * 2 * pair)


# ---- the same in plain torch, 64 bits -----------------------------------------------------------------
def _tables(L, group):
    """Dense symmetry matrices in mode space, (N_sym, n, n)."""
    s, _ = _system(L, group)
    if group != "full":
        return torch.eye(s.n_modes, dtype=F64, device=DEV)[None]
    S = torch.zeros(s.n_syms, s.n_modes, s.n_modes, dtype=F64, device=DEV)
    for blk, tab in zip(s.deg_space, s.symmetries):
        b0, b1 = int(blk[0]), int(blk[-1]) + 1
        S[:, b0:b1, b0:b1] = torch.as_tensor(tab, device=DEV)
    return S


class _Averages:
    """f = sum_ij S_j (alpha y_i + beta x~_i), D = sum_ij S_j W_ij S_j^T over every symmetry row."""

    def __init__(self, case, d):
        self.S = _tables(case["L"], case["group"])
        n = d["w"].numel()
        self.ups = 2 * d["w"] / (1 + 2 * _bose(d["w"]))
        self.mu, self.nu = torch.triu_indices(n, n, device=DEV)
        self.m = torch.where(self.mu == self.nu, 1.0, 2.0).to(F64)
        self.X, self.Y, self.rho = d["X"], d["Y"], d["rho"]
        self.pairs()

    def pairs(self):
        X, G, mu, nu = self.X, self.Y / self.ups, self.mu, self.nu
        self.G = G
        self.Q1 = X[:, mu] * X[:, nu]
        self.Q2 = X[:, mu] * G[:, nu] + X[:, nu] * G[:, mu]

    def __call__(self, R, Ys):
        n, ups, S, rho = self.ups.numel(), self.ups, self.S, self.rho
        mu, nu, X, G = self.mu, self.nu, self.X, self.G
        f = torch.zeros(n, dtype=F64, device=DEV)
        D = torch.zeros(n, n, dtype=F64, device=DEV)
        Ys = 0.5 * (Ys + Ys.T)
        for j in range(0, len(S), 512):
            Sj = S[j:j + 512]
            B = (Sj.transpose(1, 2) @ (Ys @ Sj))[:, mu, nu] * self.m
            r1 = (R @ Sj) * ups
            a, b = B @ self.Q1.T, 0.5 * (B @ self.Q2.T)
            del B
            c, e = r1 @ X.T, r1 @ G.T
            gam, dlt = rho * (a / 8 - c / 3), rho * (b / 4 - e / 3)
            Z = (gam @ self.Q2 + dlt @ self.Q1) * (ups[mu] * ups[nu])
            W = torch.zeros(len(Sj), n * n, dtype=F64, device=DEV).index_copy(1, mu * n + nu, Z).view(-1, n, n)
            W = W + W.triu(1).transpose(1, 2)
            F = -(rho * a / 6) @ self.Y - (rho * b / 3) @ (X * ups)
            f = f + (Sj @ F[:, :, None]).sum(0)[:, 0]
            D = D + ((Sj @ W) @ Sj.transpose(1, 2)).sum(0)
        norm = 1.0 / (rho.sum() * len(S))
        return f * norm, D * norm


def _apply(av, w, psi, tr, wigner):
    n, P = w.numel(), av.mu.numel()
    mu, nu = av.mu, av.nu
    na, nb = _bose(w)[mu], _bose(w)[nu]
    wa, wb = w[mu], w[nu]
    R, pY, pA = psi[:n], psi[n:n + P], psi[n + P:]
    Ya, Yb = 2 * wa / (2 * na + 1), 2 * wb / (2 * nb + 1)
    RAa, RAb = Ya * na * (na + 1), Yb * nb * (nb + 1)
    chim = (wa - wb) * (na - nb) / (2 * wa * wb)
    chip = (wa + wb) * (1 + na + nb) / (2 * wa * wb)
    sm, sp = torch.sqrt(-0.5 * chim), torch.sqrt(0.5 * chip)
    if wigner:
        w2X = 8 * wa * wb / ((1 + 2 * na) * (1 + 2 * nb))
        y = w2X * (sm * pY - sp * pA)
    elif tr:
        half = torch.where(mu == nu, 1.0, 0.5).to(F64)
        y = half * 2 * Ya * Yb * ((Ya + Yb) * pY + (RAa + RAb) * pA)
    else:
        y = pY
    Ys = torch.zeros(n, n, dtype=F64, device=DEV)
    Ys[mu, nu] = y
    Ys[nu, mu] = y
    f, D = av(R, Ys)
    d = D[mu, nu]
    if wigner:
        return torch.cat([-w * w * R + f, -(wa - wb) ** 2 * pY + sm * d, -(wa + wb) ** 2 * pA - sp * d])
    den = (2 * na + 1) * (2 * nb + 1)
    k = 2 * na * nb + na + nb
    Xab = -wa ** 2 - wb ** 2 - 2 * wa * wb / den
    Yab = -8 * wa * wb / den
    X1ab = -k * (k + 1) * 2 * wa * wb / den
    Y1ab = -wa ** 2 - wb ** 2 + 2 * wa * wb / den
    if tr:
        oY = -Xab * pY - X1ab * pA - 0.5 * d / (Ya * Yb) * av.m
        oA = -Yab * pY - Y1ab * pA
    else:
        oY = -Xab * pY - Yab * pA - d * (Ya + Yb)
        oA = -X1ab * pY - Y1ab * pA - d * (RAa + RAb)
    return torch.cat([w * w * R - f, oY, oA])


def _static(av, w, psi):
    n = w.numel()
    mu, nu = av.mu, av.nu
    y = psi[n:]
    up = -2.0 * y * av.ups[mu] * av.ups[nu]
    Ys = torch.zeros(n, n, dtype=F64, device=DEV)
    Ys[mu, nu] = up
    Ys[nu, mu] = up
    f, D = av(psi[:n], Ys)
    wb, wa, nb, na = w[mu], w[nu], _bose(w)[mu], _bose(w)[nu]
    equal = (wa - wb).abs() < 1e-8   # the reference's equal-frequency term vanishes
    diff = torch.where(equal, torch.zeros_like(wa), (na - nb) / torch.where(equal, torch.ones_like(wa), wa - wb))
    lam = ((na + nb + 1) / (wa + wb) - diff) / (4 * wa * wb)
    return torch.cat([psi[:n] * w * w - f, y / lam + D[mu, nu]])


def _chain(av, w, q0, steps):
    """The bi-conjugate recurrence of one chain: coefficients, last vectors and history."""
    q = p = q0
    qo = po = torch.zeros_like(q0)
    c1 = b1 = 0.0
    c2, s, so = 1.0, 1.0, 0.0
    coef = []
    for k in range(steps):
        Lq, pL = _apply(av, w, q, 0, False), _apply(av, w, p, 1, False)
        pn = s / (c1 if k else 1.0)
        a = float(p @ Lq) * pn
        r, t = Lq - a * q, pL - a * p
        if k:
            r = r - c1 * qo
            t = t - b1 * ((so / c2 if k > 1 else so) / pn) * po
        rn, tn = float(r.norm()), float(t.norm())
        c = float(t @ r) / tn / rn * tn * pn
        coef.append([a, rn, c, tn * pn])
        qo, po, q, p = q, p, r / rn, t / tn
        c2, so = (c1 if k else 1.0), s
        c1, b1, s = c, rn, tn * pn
    return coef, torch.stack([q, p, qo, po]), [c1, b1, s, so, c2, float(steps)]


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "green":
        sm = 5.0 / rocksalt.RY_TO_CM
        a, b, c = (d[k].cpu().numpy() for k in "abc")
        z = -d["omega"].cpu().numpy() ** 2 + 2j * d["omega"].cpu().numpy() * sm
        g = 1.0 / (a[-1] + z)
        for k in range(len(a) - 2, -1, -1):
            g = 1.0 / (a[k] + z - b[k] * c[k] * g)
        return np.stack([g.real, g.imag], axis=1).ravel()
    w = d["w"]
    if kind == "vjp":
        Y, rho = d["Y"].requires_grad_(), d["rho"].requires_grad_()
        av = _Averages(case, dict(d, Y=Y, rho=rho))
        Yb, rb = torch.zeros_like(Y), torch.zeros_like(rho)
        for k in range(case["nb"]):
            av.pairs()
            f, D = av(d["R1"][k], d["Ys"][k])
            gY, gr = torch.autograd.grad((d["fbar"][k] * f).sum() + (d["Dbar"][k] * D).sum(), (Y, rho))
            Yb, rb = Yb + gY, rb + gr
        return Yb, rb
    av = _Averages(case, d)
    if kind == "chain":
        out = [_chain(av, w, q, case["steps"]) for q in d["q"]]
        return (torch.tensor([o[0] for o in out], dtype=F64).transpose(0, 1).contiguous(),
                torch.stack([o[1] for o in out], dim=1), torch.tensor([o[2] for o in out], dtype=F64))
    if kind == "static":
        return torch.stack([_static(av, w, v) for v in d["psi"]])
    return torch.stack([_apply(av, w, v, t, case["wigner"]) for v, t in zip(d["psi"], _transpose(case["nb"]))])
