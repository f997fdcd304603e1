"""The work that users of this framework have it do, as cases to be timed.

Every case is one call (or the few calls that belong together) of the public API:
``build_fock``, ``hf_energy`` / ``free_energy``, the reverse mode (``adjoint``),
the density step of a self-consistent loop (``eigh`` -> mu -> occupations ->
density), and two whole solves.  The models are those of the repository's
benchmark and tests: a seeded Fourier Hamiltonian, gate-screened interactions
(one scalar V(q), or a layer-resolved V_ab(q)), densities U diag(f) U^H with Haar
U.  Sizes run from the 24x24 mesh of the SCF example to the 192x192 mesh of the
Fock benchmark, odd and rectangular meshes among them, with up to 16 bands.
"""

import math

import numpy as np
import torch

import jax_hf_b200 as G
from jax_hf_b200 import adjoint, linalg
from jax_hf_b200.reference_scf import SCFConfig, solve_scf
from jax_hf_b200.solver import SolverConfig, solve

# budget of the conjugate-gradient solves, in iterations
CG_ITERATIONS = 8
# iterations a DIIS solve of these models takes, for its operation count alone
SCF_ITERATIONS = 15


def _build(name, nk1, nk2, nb, V, dtype="c128", extra="none"):
    return dict(name=name, kind="build", nk1=nk1, nk2=nk2, nb=nb, V=V, dtype=dtype, extra=extra)


def listed():
    return [
        # the smallest build: the SCF example's mesh, one scalar V; launches and latency
        _build("build_24_nb4", 24, 24, 4, "scalar"),
        # odd mesh with sixteen bands, Hartree and a reference density: a moire-like model
        _build("build_49_nb16_hartree", 49, 49, 16, "scalar", extra="hartree"),
        # rectangular mesh with odd factors, six bands, contact terms too
        _build("build_90x75_nb6_contact", 90, 75, 6, "layer", extra="contact"),
        # the largest mesh of the density scan
        _build("build_120_nb8", 120, 120, 8, "layer"),
        # the headline build, in double and in single precision
        _build("build_192_nb8", 192, 192, 8, "layer"),
        _build("build_192_nb8_c64", 192, 192, 8, "layer", dtype="c64"),
        # value of the functional at a density whose Fock matrix is known (a line search's step)
        dict(name="objective_192_nb8", kind="objective", nk1=192, nk2=192, nb=8, V="layer", dtype="c128"),
        # value and gradients in the density, the occupations and the Hamiltonian
        dict(name="gradient_96_nb4", kind="gradient", nk1=96, nk2=96, nb=4, V="scalar", dtype="c128"),
        # density of a Fock matrix: eigenvectors, mu, occupations, density
        dict(name="density_49_nb16", kind="density", nk1=49, nk2=49, nb=16, T=0.5, dtype="c128"),
        dict(name="density_144_nb8", kind="density", nk1=144, nk2=144, nb=8, T=0.05, dtype="c128"),
        # whole solves: the SCF example to its tolerance, and a budget of direct minimisation
        dict(name="scf_24_nb4", kind="scf", nk1=24, nk2=24, nb=4, V="scalar", T=0.1, filling=0.5),
        dict(name="cg_144_nb8", kind="cg", nk1=144, nk2=144, nb=8, V="layer", T=0.05, filling=0.375),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: log-uniform mesh sides from 12 to 192, a third of the meshes rectangular."""
    kind = rng.choice(["build"] * 6 + ["objective"] + ["gradient"] * 2 + ["density"] * 3 + ["scf", "cg"])
    lo, hi = {"scf": (12, 48), "cg": (24, 144)}.get(kind, (12, 192))
    while True:
        n1 = _log_int(rng, lo, hi)
        n2 = _log_int(rng, lo, hi) if rng.random() < 1 / 3 else n1
        if kind in ("scf", "cg"):
            nb = rng.choice([4, 6, 8])
            break
        nb = rng.choice([2, 3, 4, 5, 6, 7, 8, 8, 12, 16])
        if kind == "density" and n1 * n2 * nb ** 3 <= 144 * 144 * 8 ** 3:
            break
        if kind != "density" and n1 * n2 * nb * nb <= 192 * 192 * 64:
            break
    V = rng.choice(["scalar", "layer"])
    if kind in ("scf", "cg"):
        return dict(kind=kind, nk1=n1, nk2=n1, nb=nb, V=V, T=0.1, filling=round(rng.uniform(0.2, 0.8), 3))
    if kind == "density":
        return dict(kind=kind, nk1=n1, nk2=n2, nb=nb, T=round(rng.uniform(0.05, 0.5), 3), dtype="c128")
    c = dict(kind=kind, nk1=n1, nk2=n2, nb=nb, V=V, dtype="c128")
    if kind == "build":
        c["dtype"] = rng.choice(["c128", "c128", "c64"])
        c["extra"] = rng.choice(["none", "none", "hartree", "contact"])
    return c


# ---------------------------------------------------------------- inputs

def _grid(n1, n2, dev):
    k1 = 2 * math.pi * (torch.arange(n1, device=dev, dtype=torch.float64) - n1 // 2) / n1
    k2 = 2 * math.pi * (torch.arange(n2, device=dev, dtype=torch.float64) - n2 // 2) / n2
    return k1[:, None].expand(n1, n2), k2[None, :].expand(n1, n2)


def _hamiltonian(rng, n1, n2, nb, dev):
    """sum_{|R| <= 2} h_R exp(i k.R), h_R complex normal over 1 + |R|^2, Hermitian."""
    k1, k2 = _grid(n1, n2, dev)
    H = torch.zeros((n1, n2, nb, nb), dtype=torch.complex128, device=dev)
    for r1 in range(-2, 3):
        for r2 in range(-2, 3):
            if r1 * r1 + r2 * r2 <= 4:
                a = (rng.standard_normal((nb, nb)) + 1j * rng.standard_normal((nb, nb))) / (1 + r1 * r1 + r2 * r2)
                ph = torch.exp(1j * (k1 * r1 + k2 * r2))
                H += ph[..., None, None] * torch.as_tensor(a, device=dev)
    return 0.5 * (H + H.mH).contiguous()


def _interaction(rng, n1, n2, nb, V, dev):
    """U 2 pi tanh(|q| d_ab) / |q| with V(0) = 0: d = 2 for the scalar V, 1 + |a - b| / 2 by layer."""
    U = rng.uniform(0.8, 1.2)
    q1, q2 = _grid(n1, n2, dev)
    q = torch.sqrt(q1 * q1 + q2 * q2)
    d = torch.full((1, 1), 2.0, dtype=torch.float64, device=dev)
    if V == "layer":
        i = torch.arange(nb, device=dev, dtype=torch.float64)
        d = 1.0 + (i[:, None] - i[None, :]).abs() / 2
    qq = torch.where(q > 0, q, torch.ones_like(q))[..., None, None]
    return torch.where(q[..., None, None] > 0, U * 2 * math.pi * torch.tanh(qq * d) / qq, torch.zeros_like(qq * d))


def _haar_density(gen, n1, n2, nb, dev):
    """U diag(f) U^H with Haar U (Gram-Schmidt of a complex normal matrix) and f uniform; also f."""
    Z = torch.randn((n1, n2, nb, nb, 2), generator=gen, device=dev, dtype=torch.float64)
    Z = torch.view_as_complex(Z)
    cols = []
    for j in range(nb):
        v = Z[..., j]
        for _ in range(2):
            for u in cols:
                v = v - u * (u.conj() * v).sum(-1, keepdim=True)
        cols.append(v / torch.linalg.vector_norm(v, dim=-1, keepdim=True))
    U = torch.stack(cols, dim=-1)
    f = torch.rand((n1, n2, nb), generator=gen, device=dev, dtype=torch.float64)
    P = (U * f[..., None, :].to(U.dtype)) @ U.mH
    return 0.5 * (P + P.mH).contiguous(), f


def _inputs(case, seed):
    """The arrays of one case in 64 bits, from the seed alone."""
    dev = torch.device("cuda", torch.cuda.current_device())
    rng = np.random.default_rng([int(seed), case["nk1"], case["nk2"], case["nb"]])
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(rng.integers(1 << 40)))
    n1, n2, nb = case["nk1"], case["nk2"], case["nb"]
    x = dict(h=_hamiltonian(rng, n1, n2, nb, dev))
    if "V" in case:
        x["V"] = _interaction(rng, n1, n2, nb, case["V"], dev)
    if case["kind"] in ("scf", "cg"):
        return x
    x["P"], x["f"] = _haar_density(gen, n1, n2, nb, dev)
    if case.get("extra", "none") != "none":
        x["ref"] = 0.5 * _haar_density(gen, n1, n2, nb, dev)[0]
        a = torch.as_tensor(rng.standard_normal((nb, nb)), device=dev)
        x["HH"] = a + a.T
    if case.get("extra") == "contact":
        O = rng.standard_normal((2, nb, nb)) + 1j * rng.standard_normal((2, nb, nb))
        x["contact"] = [(0.3, O[0], O[0].conj().T), (-0.2, O[1], O[1])]
    return x


def _complex(case):
    return torch.complex64 if case.get("dtype") == "c64" else torch.complex128


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    x = _inputs(case, seed)
    kind, n1, n2 = case["kind"], case["nk1"], case["nk2"]
    w = np.full((n1, n2), 1.0 / (n1 * n2))
    if kind == "density":
        # a Fock matrix: the Hamiltonian with an exchange-sized term of the density
        w2d = torch.as_tensor(w, device=x["h"].device)
        return dict(kind=kind, F=(x["h"] - 0.3 * x["P"]).contiguous(), w2d=w2d, T=case["T"], n=0.4375 * case["nb"])
    cdt = _complex(case)
    more = {}
    if "ref" in x:
        more = dict(include_hartree=True, reference_density=x["ref"], hartree_matrix=x["HH"],
                    contact_terms=x.get("contact"))
    T = case.get("T", 0.05)
    K = G.HartreeFockKernel(w, x["h"].to(cdt), x["V"], T, **more)
    s = dict(kind=kind, K=K)
    if kind in ("scf", "cg"):
        s["P0"] = torch.zeros_like(K.h)
        s["n"] = case["filling"] * case["nb"]
        return s
    s["P"] = x["P"].to(cdt).contiguous()
    if kind == "objective":
        s["Sigma"], s["H"], _ = _build_call(K, s["P"])
        s["p"] = x["f"]
        s["w_norm"] = K.w2d / K.weight_sum
    if kind == "gradient":
        s["p"] = x["f"]
    return s


def _build_call(K, P):
    a = K.as_args()
    return G.build_fock(P, h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"], w2d=K.w2d,
                        include_exchange=a["include_exchange"], include_hartree=a["include_hartree"],
                        exchange_hermitian_channel_packing=a["exchange_hermitian_channel_packing"],
                        contact_g=a["contact_g"], contact_Oi=a["contact_Oi"], contact_Oj=a["contact_Oj"])


def run(state):
    kind = state["kind"]
    if kind == "build":
        Sigma, H, F = _build_call(state["K"], state["P"])
        return dict(Sigma=Sigma, H=H, F=F)
    if kind == "objective":
        K = state["K"]
        E = G.hf_energy(state["P"], h=K.h, Sigma=state["Sigma"], H=state["H"], weights_b=K.weights_b)
        return dict(E=E, Omega=G.free_energy(E, state["p"], state["w_norm"], K.T))
    if kind == "gradient":
        P = state["P"].detach().requires_grad_(True)
        p = state["p"].detach().requires_grad_(True)
        h = state["K"].h.detach().requires_grad_(True)
        Omega = adjoint.objective(P, p, state["K"], h)
        Omega.backward()
        return dict(Omega=Omega.detach(), P=P.grad, p=p.grad, h=h.grad)
    if kind == "density":
        # the eigenvectors are fixed up to a phase each: the density carries them
        eps, Q = linalg.eigh(state["F"])
        mu = G.find_chemical_potential(eps, state["w2d"], state["n"], state["T"])
        p = G.fermidirac(eps - mu, state["T"])
        return dict(eps=eps, mu=mu, p=p, P=linalg.density_from_Qp(Q, p))
    if kind == "scf":
        r = solve_scf(state["K"], state["P0"], state["n"], config=SCFConfig(acceleration="diis"))
        return dict(P=r.density_matrix, F=r.fock_matrix, E=r.energy, mu=r.chemical_potential,
                    iterations=int(r.iterations))
    r = solve(state["K"], state["P0"], state["n"], config=SolverConfig(max_iter=CG_ITERATIONS, tol_E=1e-9))
    return dict(p=r.p, mu=r.mu, P=r.density, F=r.fock, E=r.energy)


# ---------------------------------------------------------------- work and the plain result

def _build_work(n1, n2, nb, e, vch, reads):
    nk, ch = n1 * n2, nb * nb
    packed = nb * (nb + 1) // 2 if vch == 1 else ch
    return (reads + 2) * nk * ch * e + nk * vch * e // 2, 2 * packed * 5 * nk * math.log2(max(nk, 2)) + 8 * nk * ch


def work(case):
    n1, n2, nb, kind = case["nk1"], case["nk2"], case["nb"], case["kind"]
    nk, ch = n1 * n2, nb * nb
    e = 8 if case.get("dtype") == "c64" else 16
    vch = ch if case.get("V") == "layer" else 1
    if kind == "build":
        b, f = _build_work(n1, n2, nb, e, vch, 2 + (case["extra"] != "none"))
    elif kind == "objective":
        b, f = 3 * nk * ch * e + nk * nb * 8, 10 * nk * ch
    elif kind == "gradient":
        b, f = _build_work(n1, n2, nb, e, vch, 2)
        b, f = b + 2 * nk * nb * 8, 2 * f + 30 * nk * ch
    else:
        # eigh: 9 n^3 complex multiply-adds; density: n^3
        step = 8 * 10 * nk * nb ** 3
        if kind == "density":
            b, f = 2 * nk * ch * e + 2 * nk * nb * 8, step
        else:
            b, f = _build_work(n1, n2, nb, 16, vch, 1)
            f = (SCF_ITERATIONS if kind == "scf" else CG_ITERATIONS) * (f + step)
    return dict(bytes=int(b), flops=int(f))


def _shifted_transform(V, w):
    """FFT2 of w V with the half-grid shift of the centred mesh taken out."""
    n1, n2 = V.shape[:2]
    ph1 = torch.exp(2j * math.pi * torch.arange(n1, device=V.device, dtype=torch.float64) * (n1 // 2) / n1)
    ph2 = torch.exp(2j * math.pi * torch.arange(n2, device=V.device, dtype=torch.float64) * (n2 // 2) / n2)
    return torch.fft.fft2((w * V).to(torch.complex128), dim=(0, 1)) * (ph1[:, None] * ph2[None, :])[..., None, None]


def _exchange(P, V, w):
    return -torch.fft.ifft2(torch.fft.fft2(P, dim=(0, 1)) * _shifted_transform(V, w), dim=(0, 1))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("scf", "cg"):
        # what an iteration returns depends on where it stops
        return None
    x = _inputs(case, seed)
    w = 1.0 / (case["nk1"] * case["nk2"])
    if kind == "density":
        return _exact_density(case, x, w)
    cdt = _complex(case)
    h, P = x["h"].to(cdt).to(torch.complex128), x["P"].to(cdt).to(torch.complex128)
    rnd = (lambda t: t.to(torch.float32).double()) if cdt == torch.complex64 else (lambda t: t)
    dP = P if "ref" not in x else P - x["ref"].to(cdt).to(torch.complex128)
    if kind == "gradient":
        P, h = P.requires_grad_(True), h.requires_grad_(True)
        dP = P
    Sigma = _exchange(dP, rnd(x["V"]), w)
    nb = case["nb"]
    H = torch.zeros((nb, nb), dtype=torch.complex128, device=h.device)
    rho = w * dP.sum((0, 1))
    if "HH" in x:
        H = torch.diag(rnd(x["HH"]) @ torch.diagonal(rho).real).to(torch.complex128)
    for g, Oi, Oj in x.get("contact", ()):
        Oi, Oj = (torch.as_tensor(O, device=h.device).to(cdt).to(torch.complex128) for O in (Oi, Oj))
        g = float(np.float32(g)) if cdt == torch.complex64 else g
        Sigma = Sigma + g * (torch.trace(Oj @ rho) * Oi - Oi @ rho @ Oj)
    if kind == "build":
        F = h + Sigma + H
        return dict(Sigma=Sigma, H=H.reshape(1, 1, nb, nb), F=0.5 * (F + F.mH))
    E = w * torch.einsum("kqab,kqba->", h + 0.5 * Sigma, P).real
    p, T = x["f"], 0.05
    if kind == "gradient":
        p = p.requires_grad_(True)
    pc = p.clamp(1e-14, 1 - 1e-14)
    Omega = E + T * w * (pc * pc.log() + (1 - pc) * torch.log1p(-pc)).sum()
    if kind == "objective":
        return dict(E=E, Omega=Omega)
    Omega.backward()
    return dict(Omega=Omega.detach(), P=P.grad, p=p.grad, h=h.grad)


def _exact_density(case, x, w):
    F = (x["h"] - 0.3 * x["P"]).cpu().numpy()
    T, n = case["T"], 0.4375 * case["nb"]
    eps, Q = np.linalg.eigh(F)

    def fermi(mu):
        return 0.5 * (1 - np.tanh((eps - mu) / (2 * (T + 1e-12))))

    lo, hi = eps.min() - 60 * T, eps.max() + 60 * T
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if w * fermi(mid).sum() < n else (lo, mid)
    mu = 0.5 * (lo + hi)
    p = fermi(mu)
    return dict(eps=eps, mu=np.float64(mu), p=p, P=(Q * p[..., None, :]) @ np.conj(np.swapaxes(Q, -1, -2)))
