"""GPU parity: CUDA Fock build / objective / per-k kernels against the CPU oracle.

Tolerances (relative to max|oracle|): complex128 1e-12 (plain FP64 target);
complex64 and the FP32-exchange mode 2e-5 (FP32 FFT round-off over <= 2*log2(N) stages).
"""

from pathlib import Path

import numpy as np
import pytest
import torch

from oracle import hf_oracle as O
from jax_hf_b200 import synthetic as S

pytestmark = pytest.mark.gpu

GOLD = Path(__file__).with_name("golden") / "meshgrid_v1.npz"
TOL64, TOL32 = 1e-12, 2e-5


def rel(a, b):
    a = a.detach().cpu().numpy() if isinstance(a, torch.Tensor) else np.asarray(a)
    b = np.asarray(b)
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def _pair(prob, dtype=np.complex128, **kw):
    import jax_hf_b200 as G
    K = G.HartreeFockKernel(prob.weights, prob.hamiltonian.astype(dtype), prob.coulomb_q, prob.T, **kw)
    Ko = O.Kernel(prob.weights, prob.hamiltonian.astype(dtype), prob.coulomb_q, prob.T, **kw)
    return K, Ko


def _fock_both(K, Ko, P, **kw):
    import jax_hf_b200 as G
    a, ao = K.as_args(), Ko.as_args()
    Sg, H, F = G.build_fock(torch.as_tensor(P, device="cuda"), h=a["h"], VR=a["VR"], refP=a["refP"],
                            HH=a["HH"], w2d=K.w2d, include_exchange=a["include_exchange"],
                            include_hartree=a["include_hartree"],
                            exchange_hermitian_channel_packing=a["exchange_hermitian_channel_packing"],
                            contact_g=a["contact_g"], contact_Oi=a["contact_Oi"], contact_Oj=a["contact_Oj"], **kw)
    So, Ho, Fo = O.build_fock(P.astype(np.complex128), h=ao["h"].astype(np.complex128), VR=ao["VR"],
                              refP=ao["refP"], HH=ao["HH"], w2d=Ko.w2d,
                              include_exchange=ao["include_exchange"], include_hartree=ao["include_hartree"],
                              exchange_hermitian_channel_packing=ao["exchange_hermitian_channel_packing"],
                              contact_g=ao["contact_g"], contact_Oi=ao["contact_Oi"], contact_Oj=ao["contact_Oj"])
    return (Sg, H, F), (So, Ho, Fo)


def test_golden_fixture(cuda):
    import jax_hf_b200 as G
    d = np.load(GOLD)
    kw = dict(include_hartree=True, include_exchange=True, reference_density=d["reference_density"].astype(np.complex128),
              hartree_matrix=d["hartree_matrix"])
    h = d["hamiltonian"].astype(np.complex128)
    K = G.HartreeFockKernel(d["weights"], h, d["coulomb_q"], float(d["T"]), **kw)
    Ko = O.Kernel(d["weights"], h, d["coulomb_q"], float(d["T"]), **kw)
    P = d["P_expected"].astype(np.complex128)
    (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P)
    assert rel(F, Fo) < TOL64
    assert rel(Sg, So) < TOL64
    assert np.abs(F.cpu().numpy() - d["F_expected"]).max() < 2e-7
    np.testing.assert_allclose(H.cpu().numpy()[0, 0], Ho[0, 0], atol=1e-14)
    E = G.hf_energy(torch.as_tensor(P, device="cuda"), h=K.h, Sigma=Sg, H=H, weights_b=K.weights_b)
    Eo = O.hf_energy(P, h=Ko.h, Sigma=So, H=Ho, weights_b=Ko.weights_b)
    assert abs(float(E) - Eo) <= 1e-12 * abs(Eo)
    assert abs(float(E) - float(d["E_expected"])) < 1e-6


def test_single_k_identity(cuda):
    """Sigma = -VR P on a 1x1 mesh (tests/test_main.py:35-41)."""
    import jax_hf_b200 as G
    P = np.array([[[[1.0 + 0.5j, 0.2], [0.2, 0.8 - 0.1j]]]])
    h = np.zeros_like(P)
    K = G.HartreeFockKernel(np.ones((1, 1)), h, np.full((1, 1, 1, 1), 0.3), 0.1)
    a = K.as_args()
    Sg, _, _ = G.build_fock(torch.as_tensor(P, device="cuda"), h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"],
                            w2d=K.w2d, include_exchange=True, include_hartree=False,
                            exchange_hermitian_channel_packing=False)
    np.testing.assert_allclose(Sg.cpu().numpy(), -0.3 * P, atol=1e-15)


CASES = [
    # nk1, nk2, nb, V, hartree/refP, contact
    (1, 1, 2, "scalar", False, False),
    (2, 3, 1, "scalar", False, False),
    (5, 7, 3, "layer", False, False),
    (12, 12, 4, "scalar", True, False),
    (24, 24, 4, "scalar", False, False),
    (36, 36, 6, "layer", False, True),
    (48, 40, 8, "layer", True, True),
    (7, 11, 5, "scalar", True, True),
    (16, 9, 8, "layer", False, False),
    (96, 96, 4, "scalar", False, False),
    (13, 26, 3, "layer", True, False),
    # band counts above the rows plan (tile slot groups / generic engine), up to the
    # largest supported nb = 32
    (10, 12, 9, "layer", True, False),
    (12, 8, 12, "scalar", False, True),
    (9, 6, 16, "layer", False, False),
    (4, 6, 32, "layer", True, False),
]


def _problem(nk1, nk2, nb, V, seed):
    rng = np.random.default_rng(seed)
    nkm = max(nk1, nk2)
    prob = S.fourier_problem(nkm, nb, 2.0, seed, V=V)
    h = prob.hamiltonian[:nk1, :nk2]
    Vq = prob.coulomb_q[:nk1, :nk2] if V == "scalar" else prob.coulomb_q[:nk1, :nk2]
    w = rng.uniform(0.5, 1.5, size=(nk1, nk2))
    w = w / w.sum()
    P = S.haar_density(nkm, nb, seed + 7)[:nk1, :nk2]
    return S.Problem("t", w, np.ascontiguousarray(h), np.ascontiguousarray(Vq), 0.1, 1.0, nkm, nb), P, rng


@pytest.mark.parametrize("nk1,nk2,nb,V,hartree,contact", CASES)
def test_fock_matches_oracle(cuda, nk1, nk2, nb, V, hartree, contact):
    prob, P, rng = _problem(nk1, nk2, nb, V, 11 + nk1 + 3 * nb)
    kw = {}
    if hartree:
        ref = S.haar_density(max(nk1, nk2), nb, 99)[:nk1, :nk2] * 0.5
        HH = rng.normal(size=(nb, nb))
        kw.update(include_hartree=True, reference_density=np.ascontiguousarray(ref), hartree_matrix=HH + HH.T)
    if contact:
        Oa = rng.normal(size=(nb, nb)) + 1j * rng.normal(size=(nb, nb))
        Ob = rng.normal(size=(nb, nb)) + 1j * rng.normal(size=(nb, nb))
        kw.update(contact_terms=[(0.3, Oa, Oa.conj().T), (-0.2, Ob, Ob)])
    K, Ko = _pair(prob, **kw)
    (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P)
    assert rel(Sg, So) < TOL64, "Sigma"
    assert rel(F, Fo) < TOL64, "F"
    # F is exactly Hermitian
    Fn = F.cpu().numpy()
    assert np.abs(Fn - np.conj(np.swapaxes(Fn, -1, -2))).max() == 0.0


def test_fock_non_hermitian_input_full_channels(cuda):
    """Layer-resolved V computes all nb^2 channels: Sigma matches the reference for any P."""
    prob, P, rng = _problem(12, 10, 4, "layer", 5)
    P = P + 0.3 * (rng.normal(size=P.shape) + 1j * rng.normal(size=P.shape))
    K, Ko = _pair(prob)
    (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P)
    assert rel(Sg, So) < TOL64 and rel(F, Fo) < TOL64


@pytest.mark.parametrize("mode", ["c64", "fp32fft"])
def test_fock_single_precision(cuda, mode):
    prob, P, _ = _problem(48, 48, 8, "layer", 3)
    if mode == "c64":
        K, Ko = _pair(prob, dtype=np.complex64)
        (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P.astype(np.complex64))
    else:
        K, Ko = _pair(prob)
        (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P, fft_precision="fp32")
        assert F.dtype == torch.complex128
    assert rel(Sg, So) < TOL32
    assert rel(F, Fo) < TOL32


def test_fock_full_size_192(cuda):
    """192x192, nb=8 layer-resolved V, Haar density: FP64 vs oracle at the benchmark size."""
    prob, P = S.fock_build_192()
    K, Ko = _pair(prob)
    (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P)
    assert rel(Sg, So) < TOL64
    assert rel(F, Fo) < TOL64
    # size-independent properties: linearity of the exchange in P
    import jax_hf_b200 as G
    a = K.as_args()
    Pt = torch.as_tensor(P, device="cuda")
    kw = dict(h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"], w2d=K.w2d, include_exchange=True,
              include_hartree=False, exchange_hermitian_channel_packing=False)
    S2, _, _ = G.build_fock(2.0 * Pt, **kw)
    assert rel(S2, 2.0 * Sg.cpu().numpy()) < 1e-14


def test_energy_entropy_free_energy(cuda):
    import jax_hf_b200 as G
    prob, P, rng = _problem(24, 20, 6, "layer", 9)
    K, Ko = _pair(prob)
    (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P)
    E = G.hf_energy(torch.as_tensor(P, device="cuda"), h=K.h, Sigma=Sg, H=H, weights_b=K.weights_b)
    Eo = O.hf_energy(P, h=Ko.h, Sigma=So, H=Ho, weights_b=Ko.weights_b)
    assert abs(float(E) - Eo) <= 1e-12 * max(abs(Eo), 1.0)
    p = rng.uniform(0, 1, size=(24, 20, 6))
    p[0, 0, 0] = 0.0
    p[0, 0, 1] = 1.0
    wn = K.w2d.cpu().numpy()
    Sent = G.occupation_entropy(torch.as_tensor(p, device="cuda"), K.w2d)
    assert abs(float(Sent) - O.occupation_entropy(p, wn)) < 1e-13
    Om = G.free_energy(E, torch.as_tensor(p, device="cuda"), K.w2d, 0.05)
    assert abs(float(Om) - O.free_energy(Eo, p, wn, 0.05)) < 1e-12 * max(1.0, abs(Eo))


@pytest.mark.parametrize("method", ["bisection", "newton"])
@pytest.mark.parametrize("T", [0.1, 0.01, 1e-5])
def test_find_mu(cuda, method, T):
    import jax_hf_b200 as G
    rng = np.random.default_rng(42)
    bands = rng.standard_normal((36, 36, 6)) * 2
    w = np.full((36, 36), 1 / 36 ** 2)
    mu = float(G.find_chemical_potential(torch.as_tensor(bands, device="cuda"), torch.as_tensor(w, device="cuda"),
                                         2.7, T, method=method))
    muo = O.find_chemical_potential(bands, w, 2.7, T, method=method)
    cnt = np.sum(w[..., None] * O.fermidirac(bands - mu, T))
    assert abs(cnt - 2.7) < 1e-9
    assert abs(mu - muo) < 1e-9 * max(1.0, abs(muo)) or T < 1e-3


@pytest.mark.parametrize("shape,T,kind", [((24, 24, 4), 0.1, "metal"), ((36, 36, 6), 0.05, "metal"),
                                          ((16, 16, 4), 0.01, "gapped"), ((12, 12, 3), 0.0, "metal"),
                                          ((96, 96, 4), 0.1, "metal")])
def test_bisection_hint_keeps_the_result(cuda, shape, T, kind):
    """hf_find_mu method 0 with a hint (mu0) decides the levels outside a certified
    bracket without evaluations; the result must be bit-identical to evaluating every
    level, for good, poor and useless hints, metals and a gapped spectrum."""
    from jax_hf_b200 import _lib
    rng = np.random.default_rng(7)
    nk1, nk2, nb = shape
    if kind == "gapped":
        lower = rng.uniform(-4, -1, (nk1, nk2, nb // 2))
        bands = np.concatenate([lower, rng.uniform(1, 4, (nk1, nk2, nb - nb // 2))], axis=-1)
        ne = float(nb // 2)
    else:
        bands = rng.standard_normal(shape) * 2
        ne = 0.4 * nb
    eps = torch.as_tensor(bands, device="cuda")
    w = torch.full((nk1, nk2), 1.0 / (nk1 * nk2), device="cuda", dtype=torch.float64)
    out = torch.zeros(1, device="cuda", dtype=torch.float64)
    L = _lib.lib()
    st = _lib.stream_ptr(eps.device)

    def run(hint):
        h = None
        if hint is not None:
            h = torch.tensor([hint], device="cuda", dtype=torch.float64)
        _lib.check(L.hf_find_mu(st, 0, 0, nk1, nk2, nb, eps.data_ptr(), w.data_ptr(), ne, T, 0,
                                None if h is None else h.data_ptr(), out.data_ptr()))
        return float(out.item())

    ref = run(None)
    if kind == "metal" and T >= 1e-3:
        # inside a gap the count is flat to rounding, and where the bisection stops there
        # depends on the summation order: only a metal's mu is compared with the oracle
        muo = O.find_chemical_potential(bands, w.cpu().numpy(), ne, T, method="bisection")
        assert abs(ref - muo) < 1e-9 * max(1.0, abs(muo))
    for hint in (ref, ref + 1e-9, ref - 1e-3, ref + 0.3, 0.0, 1e6, -50.0, float("nan")):
        assert run(hint) == ref, hint
    # the hint may alias the output (the SCF driver passes its previous mu in place)
    out.fill_(ref + 1e-6)
    _lib.check(L.hf_find_mu(st, 0, 0, nk1, nk2, nb, eps.data_ptr(), w.data_ptr(), ne, T, 0,
                            out.data_ptr(), out.data_ptr()))
    assert float(out.item()) == ref


def test_solve_mu_warm_start(cuda):
    from jax_hf_b200.utils import solve_mu
    rng = np.random.default_rng(1)
    eps = rng.standard_normal((144, 144, 8))
    w = np.full((144, 144), 1 / 144 ** 2)
    for mu0, T in ((0.0, 0.05), (0.7, 0.1), (-5.0, 0.02)):
        mu = float(solve_mu(torch.as_tensor(eps, device="cuda"), torch.as_tensor(w, device="cuda"), 3.0, mu0, T))
        muo = O.solve_mu(eps, w, 3.0, mu0, T)
        assert abs(mu - muo) < 1e-13 * max(1, abs(muo))


def test_unreachable_count_raises(cuda):
    import jax_hf_b200 as G
    with pytest.raises(ValueError, match="physically reachable range"):
        G.find_chemical_potential(torch.zeros((1, 1, 1), device="cuda", dtype=torch.float64),
                                  torch.ones((1, 1), device="cuda", dtype=torch.float64), 2.0, 0.1)


def _herm_batch(rng, shape):
    A = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    return 0.5 * (A + np.conj(np.swapaxes(A, -1, -2)))


@pytest.mark.parametrize("nb", [1, 2, 3, 4, 5, 6, 8, 12, 16])
def test_eigh(cuda, nb):
    from jax_hf_b200 import linalg as L
    rng = np.random.default_rng(nb)
    A = _herm_batch(rng, (7, 5, nb, nb))
    A[0, 0] = np.diag(np.arange(nb, dtype=float))       # already diagonal
    A[0, 1] = np.eye(nb)                                  # fully degenerate
    w, V = L.eigh(torch.as_tensor(A, device="cuda"))
    w, V = w.cpu().numpy(), V.cpu().numpy()
    wo = np.linalg.eigvalsh(A)
    assert np.abs(w - wo).max() < 1e-13 * max(1, np.abs(wo).max())
    rec = np.einsum("...in,...n,...jn->...ij", V, w, np.conj(V))
    assert np.abs(rec - A).max() < 1e-13 * max(1, np.abs(A).max())
    VhV = np.conj(np.swapaxes(V, -1, -2)) @ V
    assert np.abs(VhV - np.eye(nb)).max() < 1e-13


def test_perk_kernels(cuda):
    from jax_hf_b200 import linalg as L
    rng = np.random.default_rng(0)
    nb = 6
    d = rng.normal(size=(3, 4, nb, nb)) + 1j * rng.normal(size=(3, 4, nb, nb))
    d = 0.5 * (d - np.conj(np.swapaxes(d, -1, -2)))
    F = _herm_batch(rng, (3, 4, nb, nb))
    Q = S.haar_unitaries((3, 4), nb, rng)
    p = rng.uniform(0, 1, size=(3, 4, nb))
    t = lambda x: torch.as_tensor(x, device="cuda")
    assert rel(L.density_from_Qp(t(Q), t(p)), O.herm(O.density_from_Qp(Q, p))) < 1e-14
    assert rel(L.fock_in_orbital_basis(t(Q), t(F)), O.fock_in_orbital_basis(Q, F)) < 1e-14
    V, lam = L.cayley_spectral_setup(t(d))
    Vo, lamo = O.cayley_spectral_setup(d)
    assert np.abs(lam.cpu().numpy() - lamo).max() < 1e-13
    Fe = O.fock_in_orbital_basis(V.cpu().numpy(), F)
    for tau in (0.0, 0.3, -0.7, 1.0):
        U_lu = L.cayley_retract(t(d), tau)
        assert rel(U_lu, O.cayley_retract(d, tau)) < 1e-13
        U_sp = L.cayley_unitary_from_spectrum(V, lam, tau)
        assert rel(U_sp, O.cayley_retract(d, tau)) < 1e-12
        dg = L.diag_UFU_from_spectrum(V, t(Fe), lam, tau)
        U = O.cayley_retract(d, tau)
        ref = np.real(np.diagonal(np.conj(np.swapaxes(U, -1, -2)) @ F @ U, axis1=-2, axis2=-1))
        assert np.abs(dg.cpu().numpy() - ref).max() < 1e-12
        assert rel(L.qr_retract(t(d), tau), O.qr_retract(d, tau)) < 1e-12


FAST_N = [12, 16, 24, 32, 36, 48, 64, 72, 96, 128, 144, 192]


@pytest.mark.parametrize("n1,n2", [(n, n) for n in FAST_N] + [(24, 48), (192, 144), (12, 36)])
@pytest.mark.parametrize("nb,V", [(1, "scalar"), (3, "layer"), (4, "scalar"), (8, "layer")])
def test_fast_engine_matches_generic(cuda, n1, n2, nb, V):
    """Register-FFT passes of the specialised mesh lengths == generic Stockham engine."""
    import jax_hf_b200 as G
    if n1 * n2 * nb * nb > 192 * 192 * 16 and nb == 8 and (n1, n2) != (192, 192):
        pytest.skip("size covered by the 192 case")
    prob, P, rng = _problem(n1, n2, nb, V, 31 + n1 + nb)
    K = G.HartreeFockKernel(prob.weights, prob.hamiltonian, prob.coulomb_q, prob.T)
    a = K.as_args()
    Pt = torch.as_tensor(P, device="cuda")
    kw = dict(h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"], w2d=K.w2d, include_exchange=True,
              include_hartree=False, exchange_hermitian_channel_packing=a["exchange_hermitian_channel_packing"])
    Sf, _, Ff = G.build_fock(Pt, **kw)
    Sg, _, Fg = G.build_fock(Pt, engine="generic", **kw)
    assert rel(Sf, Sg.cpu().numpy()) < TOL64
    assert rel(Ff, Fg.cpu().numpy()) < TOL64
    Sm, _, Fm = G.build_fock(Pt, fft_precision="fp32", **kw)
    assert rel(Sm, Sg.cpu().numpy()) < TOL32
    St, _, Ft = G.build_fock(Pt, engine="tile", **kw)  # 2x2-tile slot groups instead of the rows plan
    assert rel(St, Sg.cpu().numpy()) < TOL64
    assert rel(Ft, Fg.cpu().numpy()) < TOL64


@pytest.mark.parametrize("n1,n2,nb,V,hartree", [(48, 48, 8, "layer", False), (36, 36, 6, "layer", True),
                                                (24, 24, 4, "scalar", False), (30, 30, 8, "layer", False)])
def test_autotune_picks_a_schedule_that_matches(cuda, n1, n2, nb, V, hartree):
    """hf_fock_autotune: every candidate timed, outputs equal the default build, choice reused."""
    import jax_hf_b200 as G
    from jax_hf_b200 import fock as Fk
    prob, P, rng = _problem(n1, n2, nb, V, 7 + n1 + nb)
    hk = dict(include_hartree=True, hartree_matrix=0.2 + 0.5 * np.eye(nb),
              reference_density=0.3 * P) if hartree else {}
    K = G.HartreeFockKernel(prob.weights, prob.hamiltonian, prob.coulomb_q, prob.T, **hk)
    a = K.as_args()
    Pt = torch.as_tensor(P, device="cuda")
    kw = dict(h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"], w2d=K.w2d, include_exchange=True,
              include_hartree=hartree, exchange_hermitian_channel_packing=a["exchange_hermitian_channel_packing"])
    Fk.autotune_reset()
    S0, H0, F0 = G.build_fock(Pt, **kw)
    try:
        S1, H1, F1 = G.build_fock(Pt, autotune=True, autotune_reps=2, **kw)
        info = dict(Fk.last_autotune)
        assert info["shape"] == (n1, n2, nb)
        assert info["chosen"] in info["us"] and all(v > 0 for v in info["us"].values())
        assert "generic" in info["us"] and "default" in info["us"]
        assert rel(S1, S0.cpu().numpy()) < TOL64 and rel(F1, F0.cpu().numpy()) < TOL64
        assert rel(H1, H0.cpu().numpy()) < TOL64
        S2, _, F2 = G.build_fock(Pt, **kw)  # the stored choice
        assert rel(S2, S0.cpu().numpy()) < TOL64 and rel(F2, F0.cpu().numpy()) < TOL64
    finally:
        Fk.autotune_reset()


SYM_CASES = [
    (48, 48, 8, False, False, None),
    (24, 36, 6, True, True, None),
    (20, 14, 5, False, False, None),          # generic engine lengths
    (48, 48, 8, False, False, "fp32"),
    (48, 48, 8, False, False, "c64"),
    (36, 36, 4, False, False, "generic"),
]


@pytest.mark.parametrize("nk1,nk2,nb,hartree,contact,mode", SYM_CASES)
def test_fock_hermitian_density_packing_band_resolved(cuda, nk1, nk2, nb, hartree, contact, mode):
    """hermitian_density=True with a real, pair-symmetric band-resolved V transforms only the
    upper-triangle channels; for a Hermitian density the result equals the full reference build."""
    prob, P, rng = _problem(nk1, nk2, nb, "layer", 17 + nk1 + nb)
    kw = {}
    if hartree:
        ref = S.haar_density(max(nk1, nk2), nb, 98)[:nk1, :nk2] * 0.5
        HH = rng.normal(size=(nb, nb))
        kw.update(include_hartree=True, reference_density=np.ascontiguousarray(ref), hartree_matrix=HH + HH.T)
    if contact:
        Oa = rng.normal(size=(nb, nb)) + 1j * rng.normal(size=(nb, nb))
        kw.update(contact_terms=[(0.3, Oa, Oa.conj().T)])
    dtype = np.complex64 if mode == "c64" else np.complex128
    K, Ko = _pair(prob, dtype=dtype, **kw)
    assert K.v_pair_symmetric
    extra = {"hermitian_density": True}
    if mode == "fp32":
        extra["fft_precision"] = "fp32"
    if mode == "generic":
        extra["engine"] = "generic"
    (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P.astype(dtype), **extra)
    tol = TOL32 if mode in ("fp32", "c64") else TOL64
    assert rel(Sg, So) < tol, "Sigma"
    assert rel(F, Fo) < tol, "F"
    Fn = F.cpu().numpy()
    assert np.abs(Fn - np.conj(np.swapaxes(Fn, -1, -2))).max() == 0.0


def test_fock_hermitian_density_packing_192(cuda):
    """The benchmark workload (192x192, nb=8, layer V, Haar density) through the packed path."""
    prob, P = S.fock_build_192()
    K, Ko = _pair(prob)
    (Sg, H, F), (So, Ho, Fo) = _fock_both(K, Ko, P, hermitian_density=True)
    assert rel(Sg, So) < TOL64
    assert rel(F, Fo) < TOL64



@pytest.mark.parametrize("streams", [1, 2, 3])
def test_build_fock_batch_matches_single_calls(cuda, streams):
    """Independent builds spread over internal streams (each with its own scratch) give
    exactly the single-call results; ``outs`` are filled in place."""
    import jax_hf_b200 as G
    prob, P, rng = _problem(48, 40, 8, "layer", 23)
    HH = rng.normal(size=(8, 8))
    ref = S.haar_density(48, 8, 5)[:48, :40] * 0.5
    K, _ = _pair(prob, include_hartree=True, reference_density=np.ascontiguousarray(ref), hartree_matrix=HH + HH.T)
    a = K.as_args()
    kw = dict(h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"], w2d=K.w2d, include_exchange=True,
              include_hartree=True, exchange_hermitian_channel_packing=a["exchange_hermitian_channel_packing"],
              contact_g=a["contact_g"], contact_Oi=a["contact_Oi"], contact_Oj=a["contact_Oj"])
    Ps = [torch.as_tensor(np.ascontiguousarray(S.haar_density(48, 8, 40 + i)[:48, :40]), device="cuda")
          for i in range(5)]
    single = [G.build_fock(Pi, **kw) for Pi in Ps]
    outs = [tuple(torch.full_like(x, float("nan")) for x in r) for r in single]
    got = G.build_fock_batch(Ps, outs=outs, streams=streams, **kw)
    torch.cuda.synchronize()
    for (s1, h1, f1), (s2, h2, f2), o in zip(single, got, outs):
        assert torch.equal(s1, s2) and torch.equal(h1, h2) and torch.equal(f1, f2)
        assert s2.data_ptr() == o[0].data_ptr() and f2.data_ptr() == o[2].data_ptr()
    # without outs, and numpy inputs
    got2 = G.build_fock_batch([Pi.cpu().numpy() for Pi in Ps], streams=streams, **kw)
    for (s1, _, f1), (s2, _, f2) in zip(single, got2):
        assert torch.equal(s1, s2) and torch.equal(f1, f2)
    with pytest.raises(ValueError, match="outs has"):
        G.build_fock_batch(Ps, outs=outs[:2], **kw)


@pytest.mark.parametrize("nb", [2, 3, 4, 5, 8, 9, 13, 16, 17])
@pytest.mark.parametrize("nk,dt", [(1, np.complex128), (33, np.complex128), (300, np.complex64)])
def test_eigh_shapes_scales_and_clusters(cuda, nb, nk, dt):
    """hf_eigh over the lane groups and the CTA remainders: random, diagonal, block-split, clustered,
    zero, huge and tiny matrices.  Backward error and orthogonality within 30 nb ulp (n sweeps of
    n rotations and n reflections, each a few ulp), eigenvalues within the same of ||A||."""
    from jax_hf_b200 import linalg as L
    rng = np.random.default_rng(nb * nk)
    A = _herm_batch(rng, (nk, nb, nb))
    special = [np.zeros((nb, nb)), np.diag(np.arange(nb)[::-1] - 1.0), 2.0 * np.eye(nb) + 1e-13 * A[0],
               np.kron(np.eye(nb // 2 + 1), np.array([[0, 1], [1, 0]]))[:nb, :nb], 1e30 * A[0], 1e-30 * A[0],
               np.ones((nb, nb))]
    for i, M in enumerate(special[:nk - 1]):
        A[1 + i] = M
    A = A.astype(dt)
    w, V = L.eigh(torch.as_tensor(A, device="cuda"))
    w, V = w.cpu().numpy().astype(np.float64), V.cpu().numpy().astype(np.complex128)
    A = A.astype(np.complex128)
    tol = 30 * nb * (2.2e-16 if dt == np.complex128 else 1.2e-7)
    nrm = np.maximum(np.linalg.norm(A, 2, axis=(-2, -1)), 1e-300)
    assert (np.diff(w, axis=-1) >= 0).all()
    assert (np.abs(w - np.linalg.eigvalsh(A)).max(-1) <= tol * nrm).all()
    rec = np.einsum("kin,kn,kjn->kij", V, w, np.conj(V))
    assert (np.abs(rec - A).max((-2, -1)) <= tol * nrm).all()
    assert np.abs(np.conj(np.swapaxes(V, -1, -2)) @ V - np.eye(nb)).max() <= tol


def test_eigh_non_finite_entries_stay_in_their_matrix(cuda):
    from jax_hf_b200 import linalg as L
    A = _herm_batch(np.random.default_rng(3), (9, 6, 6))
    A[2, 1, 4] = np.nan
    A[5, 0, 0] = np.inf
    w, V = L.eigh(torch.as_tensor(A, device="cuda"))
    bad = torch.tensor([2, 5], device="cuda")
    assert torch.isnan(w[bad]).all() and torch.isnan(V[bad].real).all()
    good = [i for i in range(9) if i not in (2, 5)]
    wo = np.linalg.eigvalsh(A[good])
    assert np.abs(w.cpu().numpy()[good] - wo).max() < 1e-13 * np.abs(wo).max()


TWO_FACTOR = [  # sides: prime radices, one-factor sides, unequal factors, the largest, mixed with a register side
    (13, 13, 3, "layer", "c128"), (1, 30, 2, "scalar", "c128"), (14, 22, 8, "layer", "c128"),
    (25, 49, 16, "scalar", "c128"), (75, 90, 6, "layer", "c128"), (48, 45, 5, "layer", "c128"),
    (120, 20, 8, "layer", "c64"), (26, 169, 4, "scalar", "c64"), (256, 10, 1, "layer", "c128"),
    (60, 27, 8, "layer", "fp32fft"), (208, 15, 9, "scalar", "c128"), (121, 21, 7, "layer", "c128"),
]


@pytest.mark.parametrize("n1,n2,nb,V,mode", TWO_FACTOR)
@pytest.mark.parametrize("terms", [False, True])
def test_two_factor_passes_match_stockham(cuda, n1, n2, nb, V, mode, terms, register_side=False):
    """Sides with two factors of at most 16 against the Stockham engine on the same inputs (FP64: both
    within 1e-12 of the oracle, so within 2e-12 of each other; FP32 transforms: 2 x 2e-5), with and
    without the reference density, Hartree and contact terms, for a density that is not Hermitian
    when every channel is transformed."""
    import jax_hf_b200 as G
    rng = np.random.default_rng(n1 + 3 * n2 + nb)
    q = lambda *s: rng.normal(size=s) + 1j * rng.normal(size=s)
    h = q(n1, n2, nb, nb)
    h = h + np.conj(np.swapaxes(h, -1, -2))
    P = q(n1, n2, nb, nb)
    if V == "scalar":
        P = 0.5 * (P + np.conj(np.swapaxes(P, -1, -2)))
    Vq = rng.uniform(0.1, 1.0, size=(n1, n2) + ((1, 1) if V == "scalar" else (nb, nb)))
    kw = {}
    if terms:
        HH = rng.normal(size=(nb, nb))
        ref = q(n1, n2, nb, nb)
        kw = dict(include_hartree=True, hartree_matrix=HH + HH.T, contact_terms=[(0.3, q(nb, nb), q(nb, nb))] * 2,
                  reference_density=0.25 * (ref + np.conj(np.swapaxes(ref, -1, -2))))
    dt = np.complex64 if mode == "c64" else np.complex128
    w = rng.uniform(0.5, 1.5, size=(n1, n2)) / (n1 * n2)
    K = G.HartreeFockKernel(w, h.astype(dt), Vq, 0.1, **kw)
    a = K.as_args()
    run = lambda **e: G.build_fock(
        torch.as_tensor(P.astype(dt), device="cuda"), h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"], w2d=K.w2d,
        include_exchange=True, include_hartree=a["include_hartree"],
        exchange_hermitian_channel_packing=a["exchange_hermitian_channel_packing"], contact_g=a["contact_g"],
        contact_Oi=a["contact_Oi"], contact_Oj=a["contact_Oj"],
        fft_precision="fp32" if mode == "fp32fft" else None, **e)
    tol = 2 * (TOL64 if mode == "c128" else TOL32)
    for x, y in zip(run(), run(engine="generic")):
        assert rel(x, y.cpu().numpy()) < tol if y.abs().max() > 0 else torch.equal(x, y)
    for x, y in zip(run(engine="stockham"), run(engine="generic")):  # the register passes at their sides
        assert register_side or torch.equal(x, y)


DENSE = [  # sides with a prime factor of 17 or more: one row, several rows, an even N2, both sides, the largest
    (17, 17, 3, "layer", "c128"), (34, 37, 8, "layer", "c128"), (61, 24, 4, "scalar", "c64"),
    (191, 3, 2, "layer", "c128"), (74, 19, 6, "layer", "fp32fft"), (12, 97, 8, "layer", "c128"),
    (306, 4, 1, "layer", "c128"), (5, 430, 2, "scalar", "c128"), (23, 29, 16, "scalar", "c128"),
]


@pytest.mark.parametrize("n1,n2,nb,V,mode", DENSE)
@pytest.mark.parametrize("terms", [False, True])
def test_dense_line_sums_match_stockham(cuda, n1, n2, nb, V, mode, terms):
    test_two_factor_passes_match_stockham(cuda, n1, n2, nb, V, mode, terms)


DEEP = [  # register sides that the slot tiles leave to the two-factor passes, and one that keeps the pair on the other
    (96, 96, 4, "scalar", "c128"), (96, 192, 9, "layer", "c64"), (192, 96, 3, "scalar", "fp32fft"),
    (192, 128, 4, "scalar", "c128"),
]


@pytest.mark.parametrize("n1,n2,nb,V,mode", DEEP)
@pytest.mark.parametrize("terms", [False, True])
def test_slot_tiles_of_deep_line_shapes_match_stockham(cuda, n1, n2, nb, V, mode, terms):
    test_two_factor_passes_match_stockham(cuda, n1, n2, nb, V, mode, terms, register_side=True)


@pytest.mark.parametrize("shape,T,kind", [((70, 59, 4), 0.1, "metal"), ((128, 128, 1), 0.02, "metal"),
                                          ((96, 96, 4), 1e-4, "metal"), ((64, 64, 8), 0.01, "gapped"),
                                          ((80, 80, 3), 0.0, "metal"), ((144, 144, 8), 0.05, "metal")])
@pytest.mark.parametrize("fill", [0.01, 0.43, 0.5, 1.0])
def test_grid_wide_mu_equals_the_cluster_bisection(cuda, shape, T, kind, fill):
    """hf_find_mu_ws (certifying passes over the grid) against hf_find_mu on the same eigenvalues: the
    bisection bit for bit; the Newton rule's root within the noise of the count (sum of n terms,
    (n / threads + 40) ulp of the total weight over N') or, where N' vanishes, the same count."""
    from jax_hf_b200 import _lib
    rng = np.random.default_rng(shape[0] + shape[2])
    eps = rng.normal(size=shape)
    if kind == "gapped":
        eps += 3.0 * np.sign(np.arange(shape[2]) - shape[2] / 2 + 0.5)
    w = rng.uniform(0.5, 1.5, size=shape[:2])
    w /= w.sum()
    nb, nk = shape[2], shape[0] * shape[1]
    e, wt = torch.as_tensor(eps, device="cuda").contiguous(), torch.as_tensor(w, device="cuda")
    L = _lib.lib()
    n = _lib.C.c_size_t(0)
    _lib.check(L.hf_mu_workspace_size(_lib.C.byref(n)))
    ws = torch.full((n.value,), 255, dtype=torch.uint8, device="cuda")
    mu0 = torch.tensor(0.1, dtype=torch.float64, device="cuda")
    out = torch.empty(4, dtype=torch.float64, device="cuda")
    s = _lib.stream_ptr(e.device)
    ne = fill * nb
    for i, (meth, m0) in enumerate(((0, None), (2, mu0.data_ptr()))):
        _lib.check(L.hf_find_mu(s, _lib.HF_C128, meth, nk, 1, nb, e.data_ptr(), wt.data_ptr(), ne, T, 0, m0,
                                out[2 * i:].data_ptr()))
        _lib.check(L.hf_find_mu_ws(s, _lib.HF_C128, meth, nk, 1, nb, e.data_ptr(), wt.data_ptr(), ne, T, 0, m0,
                                   out[2 * i + 1:].data_ptr(), ws.data_ptr(), ws.numel()))
    mu = out.cpu().numpy()
    assert mu[0] == mu[1]
    count = lambda m: float((w[..., None] / (1.0 + np.exp(np.clip((eps - m) / max(T, 1e-12), -700, 700)))).sum())
    if abs(mu[2] - mu[3]) > 1e-11 * max(1.0, abs(mu[2])):
        assert abs(count(mu[2]) - count(mu[3])) <= 60 * 2.2e-16 * nb


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("method", [0, 2])
def test_grid_wide_mu_with_a_non_finite_eigenvalue(cuda, method, bad):
    """A non-finite eigenvalue drives hf_find_mu_ws to the bits of hf_find_mu (the certifying passes must not
    take a NaN for an empty state)."""
    from jax_hf_b200 import _lib
    rng = np.random.default_rng(5)
    nk, nb = 128 * 128, 8
    eps = rng.normal(size=(nk, nb))
    eps[1234, 2] = bad
    e, w = torch.as_tensor(eps, device="cuda"), torch.full((nk,), 1.0 / nk, dtype=torch.float64, device="cuda")
    L = _lib.lib()
    n = _lib.C.c_size_t(0)
    _lib.check(L.hf_mu_workspace_size(_lib.C.byref(n)))
    ws = torch.full((n.value,), 255, dtype=torch.uint8, device="cuda")
    mu0 = torch.tensor(0.1, dtype=torch.float64, device="cuda")
    m0 = mu0.data_ptr() if method else None
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    s = _lib.stream_ptr(e.device)
    _lib.check(L.hf_find_mu(s, _lib.HF_C128, method, nk, 1, nb, e.data_ptr(), w.data_ptr(), 1.7, 0.1, 0, m0, out.data_ptr()))
    _lib.check(L.hf_find_mu_ws(s, _lib.HF_C128, method, nk, 1, nb, e.data_ptr(), w.data_ptr(), 1.7, 0.1, 0, m0,
                               out[1:].data_ptr(), ws.data_ptr(), ws.numel()))
    assert torch.equal(out[:1], out[1:]) or torch.isnan(out).all()


@pytest.mark.parametrize("nb", [2, 7, 8, 9, 13, 16, 17])
@pytest.mark.parametrize("nk,dt", [(1, np.complex128), (37, np.complex64), (130, np.complex128)])
def test_density_from_orbitals_shapes(cuda, nb, nk, dt):
    """P = herm(Q diag(p) Q^H) over the lane groups and CTA remainders: nb products of numbers of
    modulus <= 1, so 4 nb ulp of the storage precision."""
    from jax_hf_b200 import linalg as L
    rng = np.random.default_rng(nb + nk)
    Q = S.haar_unitaries((nk,), nb, rng).astype(dt)
    p = rng.uniform(0, 1, size=(nk, nb)).astype(np.zeros(1, dt).real.dtype)
    P = L.density_from_Qp(torch.as_tensor(Q, device="cuda"), torch.as_tensor(p, device="cuda")).cpu().numpy()
    ref = np.einsum("kin,kn,kjn->kij", Q.astype(np.complex128), p.astype(float), np.conj(Q.astype(np.complex128)))
    assert np.abs(P - ref).max() <= 4 * nb * (1.2e-7 if dt == np.complex64 else 2.3e-16)
    assert np.abs(P - np.conj(np.swapaxes(P, -1, -2))).max() == 0.0


@pytest.mark.parametrize("T", [0.05, 1e-4])
def test_find_mu_from_two_threads_on_one_stream(cuda, T):
    """Two threads that find the mu of their own spectra on the same stream get what one thread gets."""
    import threading

    import jax_hf_b200 as G
    from jax_hf_b200.utils import solve_mu
    g = torch.Generator(device="cuda").manual_seed(2)
    w = torch.full((128 * 200,), 1.0 / (128 * 200), dtype=torch.float64, device="cuda")
    eps = [i + torch.randn(128 * 200, 8, dtype=torch.float64, device="cuda", generator=g) for i in range(2)]
    call = (lambda e: float(G.find_chemical_potential(e, w, 2.7, T)), lambda e: float(solve_mu(e, w, 2.7, 0.3, T)))
    for f in call:
        want = [f(e) for e in eps]
        got = [[], []]
        threads = [threading.Thread(target=lambda i=i: got[i].extend(f(eps[i]) for _ in range(60))) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for i in range(2):
            assert got[i] == [want[i]] * 60


def _tune_inputs(n, nb, V):
    import jax_hf_b200 as G
    prob, P, _ = _problem(n, n, nb, V, 3)
    K = G.HartreeFockKernel(prob.weights, prob.hamiltonian, prob.coulomb_q, prob.T)
    a = K.as_args()
    return torch.as_tensor(P, device="cuda"), dict(
        h=a["h"], VR=a["VR"], refP=a["refP"], HH=a["HH"], w2d=K.w2d, include_exchange=True, include_hartree=False,
        exchange_hermitian_channel_packing=a["exchange_hermitian_channel_packing"])


def test_autotuning_the_stockham_stages_leaves_other_builds_alone(cuda):
    """Tuned with engine="stockham", a two-factor side compares two schedules of the Stockham stages; whichever
    wins, the default build keeps the two-factor passes (the same bits as before), and a build tuned by
    default leaves the Stockham one where it was."""
    import jax_hf_b200 as G
    from jax_hf_b200 import fock as Fk
    P, kw = _tune_inputs(60, 3, "layer")
    Fk.autotune_reset()
    try:
        before = G.build_fock(P, **kw)
        for _ in range(20):  # two equal candidates: the noise of the timing picks one
            G.build_fock(P, engine="stockham", autotune=True, autotune_reps=1, **kw)
            if Fk.last_autotune["chosen"] == "generic":
                break
        after = G.build_fock(P, **kw)
        assert all(torch.equal(x, y) for x, y in zip(before, after))
    finally:
        Fk.autotune_reset()


def test_autotuner_times_the_register_passes_beside_the_two_factor_ones(cuda):
    """96 x 96 packed runs the two-factor passes by default: the tile candidate is the register passes."""
    import jax_hf_b200 as G
    from jax_hf_b200 import fock as Fk
    P, kw = _tune_inputs(96, 4, "scalar")
    Fk.autotune_reset()
    try:
        G.build_fock(P, autotune=True, autotune_reps=1, **kw)
        assert Fk.last_autotune["us"]["tile"] > 0 and "pipe" not in Fk.last_autotune["us"]
        G.build_fock(P, engine="stockham", autotune=True, autotune_reps=1, **kw)
        assert "tile" not in Fk.last_autotune["us"]
    finally:
        Fk.autotune_reset()


@pytest.mark.parametrize("center,width,T", [(10.0, 0.02, 1e-3), (10.0, 0.02, 1e-2), (1.0, 0.002, 1e-3),
                                            (-300.0, 0.5, 1e-2), (1e4, 0.1, 0.05), (0.0, 1.0, 1e-3)])
@pytest.mark.parametrize("nk", [576, 10368])
def test_bisection_hint_keeps_the_result_of_narrow_bands(cuda, center, width, T, nk):
    """Bands that are narrow against their offset from zero, where the spacing of the numbers at mu exceeds what
    the certifying margin is worth: with a hint the result still has the bits of evaluating every level."""
    from jax_hf_b200 import _lib
    rng = np.random.default_rng(nk)
    eps = torch.as_tensor(center + width * rng.standard_normal((nk, 4)), device="cuda")
    w = torch.full((nk,), 1.0 / nk, device="cuda", dtype=torch.float64)
    fills = rng.uniform(0.05, 3.95, 60)
    L, st = _lib.lib(), _lib.stream_ptr(eps.device)
    out = torch.zeros(4, len(fills), device="cuda", dtype=torch.float64)
    hint = torch.zeros(3, len(fills), device="cuda", dtype=torch.float64)

    def run(ne, h, o):
        _lib.check(L.hf_find_mu(st, _lib.HF_C128, 0, nk, 1, 4, eps.data_ptr(), w.data_ptr(), ne, T, 0, h, o))

    for i, ne in enumerate(fills):
        run(ne, None, out[0, i:].data_ptr())
    hint.copy_(out[0] + width * torch.tensor([[1e-8], [1e-4], [-0.3]], device="cuda"))
    for j in range(3):
        for i, ne in enumerate(fills):
            run(ne, hint[j, i:].data_ptr(), out[j + 1, i:].data_ptr())
    for j in range(1, 4):
        assert torch.equal(out[j], out[0]), (out[j] != out[0]).sum()


@pytest.mark.parametrize("T", [0.3, 0.02, -0.05])
def test_grid_wide_bisection_where_the_count_is_not_monotonic(cuda, T):
    """Weights of both signs (quadrature rules have them) and T < 0: no bracket can be certified there, so
    hf_find_mu_ws evaluates the levels that hf_find_mu evaluates."""
    from jax_hf_b200 import _lib
    rng = np.random.default_rng(8)
    nk, nb = 96 * 96, 4
    bands, wn = rng.normal(size=(nk, nb)), np.ones(nk)
    if T > 0:  # the count falls where the negative weights' eigenvalues lie
        wn[::4] = -1.5
        bands[::4] = 0.4 + 0.1 * bands[::4]
    eps = torch.as_tensor(bands, device="cuda")
    w = torch.as_tensor(wn / wn.sum(), device="cuda")
    L, st = _lib.lib(), _lib.stream_ptr(eps.device)
    n = _lib.C.c_size_t(0)
    _lib.check(L.hf_mu_workspace_size(_lib.C.byref(n)))
    ws = torch.full((n.value,), 255, dtype=torch.uint8, device="cuda")
    fills = np.linspace(-0.2, nb + 0.2, 81)
    out = torch.zeros(2, len(fills), dtype=torch.float64, device="cuda")
    for i, ne in enumerate(fills):
        args = (st, _lib.HF_C128, 0, nk, 1, nb, eps.data_ptr(), w.data_ptr(), ne, T, 0, None)
        _lib.check(L.hf_find_mu(*args, out[0, i:].data_ptr()))
        _lib.check(L.hf_find_mu_ws(*args, out[1, i:].data_ptr(), ws.data_ptr(), ws.numel()))
    assert torch.equal(out[0], out[1])


def _fma(x, y, z):
    from fractions import Fraction
    return float(Fraction(x) * Fraction(y) + Fraction(z))


@pytest.mark.parametrize("n,nb", [(5, 3), (90, 6), (49, 16), (144, 2), (40, 8)])
@pytest.mark.parametrize("packing", [False, True])
def test_constant_terms_add_the_rows_one_by_one(cuda, n, nb, packing):
    """The constant terms of a build keep the roundings of adding the mesh rows in order (an SCF loop's DIIS
    amplifies any other order).  One k-point per row and weight 1 make a row's partial sum P itself, and the
    identity as Hartree matrix makes H its running sum, so plain sequential sums are the oracle, bit for bit."""
    import jax_hf_b200 as G
    rng = np.random.default_rng(n + nb)
    P = rng.normal(size=(n, 1, nb, nb)) + 1j * rng.normal(size=(n, 1, nb, nb))
    P = 0.5 * (P + np.conj(np.swapaxes(P, -1, -2)))
    t = lambda x: torch.as_tensor(x, device="cuda")
    VR = t(np.ones((n, 1, 1, 1)))
    _, H, _ = G.build_fock(t(P), h=t(np.zeros_like(P)), VR=VR, refP=None, HH=t(np.eye(nb)), w2d=t(np.ones((n, 1))),
                           include_exchange=packing, include_hartree=True, exchange_hermitian_channel_packing=packing)
    s = np.zeros(nb)
    for k in range(n):
        s = s + np.einsum("aa->a", P[k, 0]).real
    assert np.array_equal(np.einsum("aa->a", H.cpu().numpy()[0, 0]).real, s)


@pytest.mark.parametrize("nb", [1, 3, 8])
def test_contact_term_keeps_its_roundings(cuda, nb):
    """Sigma of one contact term at one k-point against the same sums in exact fused multiply-adds: products
    a.x b.x - a.y b.y and a.x b.y + a.y b.x with one fused rounding each, added to the running sum."""
    import jax_hf_b200 as G
    rng = np.random.default_rng(nb)
    P, Oi, Oj = (rng.normal(size=(nb, nb)) + 1j * rng.normal(size=(nb, nb)) for _ in range(3))
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device="cuda")
    S, _, _ = G.build_fock(t(P[None, None]), h=t(np.zeros((1, 1, nb, nb), complex)), VR=None, refP=None,
                           HH=t(np.zeros((nb, nb))), w2d=t(np.ones((1, 1))), include_exchange=False,
                           include_hartree=True, exchange_hermitian_channel_packing=False,
                           contact_g=t(np.array([1.0])), contact_Oi=t(Oi[None]), contact_Oj=t(Oj[None]))
    prod = lambda a, b: complex(_fma(a.real, b.real, -(a.imag * b.imag)), _fma(a.imag, b.real, a.real * b.imag))

    def dot(pairs):
        z = 0j
        for a, b in pairs:
            z = z + prod(complex(a), complex(b))
        return z

    tr = dot([(Oj[a, b], P[b, a]) for a in range(nb) for b in range(nb)])
    R = [[dot([(Oi[i, k], P[k, l]) for k in range(nb)]) for l in range(nb)] for i in range(nb)]
    for i in range(nb):
        for l in range(nb):
            o = complex(Oi[i, l])
            ht = complex(_fma(o.real, tr.real, -(o.imag * tr.imag)), _fma(o.real, tr.imag, o.imag * tr.real))
            assert complex(S[0, 0, i, l].item()) == ht - dot([(R[i][k], Oj[k, l]) for k in range(nb)])


@pytest.mark.parametrize("nb,dt", [(9, np.complex128), (12, np.complex128), (16, np.complex128), (3, np.complex64),
                                   (8, np.complex64), (13, np.complex64)])
@pytest.mark.parametrize("nk", [1, 45])
def test_density_from_orbitals_has_the_bits_of_the_general_kernel(cuda, nb, dt, nk):
    """The column kernel against the warp-per-matrix kernel, which takes the same orbitals padded with zeros
    to 17 bands: the padding adds zeros to sums in the same order, so the bits are the same."""
    from jax_hf_b200 import linalg as L
    rng = np.random.default_rng(nb + nk)
    Q = (rng.normal(size=(nk, nb, nb)) + 1j * rng.normal(size=(nk, nb, nb))).astype(dt)
    p = rng.uniform(0, 1, size=(nk, nb)).astype(np.zeros(1, dt).real.dtype)
    Qp, pp = np.zeros((nk, 17, 17), dt), np.zeros((nk, 17), p.dtype)
    Qp[:, :nb, :nb], pp[:, :nb] = Q, p
    t = lambda x: torch.as_tensor(x, device="cuda")
    assert torch.equal(L.density_from_Qp(t(Q), t(p)), L.density_from_Qp(t(Qp), t(pp))[:, :nb, :nb])


def _mu_pair(eps, w, ne, T, method, mu0, maxiter=0):
    """hf_find_mu and hf_find_mu_ws (a dirty workspace) on the same eigenvalues."""
    from jax_hf_b200 import _lib
    L, s = _lib.lib(), _lib.stream_ptr(eps.device)
    n = _lib.C.c_size_t(0)
    _lib.check(L.hf_mu_workspace_size(_lib.C.byref(n)))
    ws = torch.full((n.value,), 255, dtype=torch.uint8, device="cuda")
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    m0 = None if mu0 is None else torch.tensor(mu0, dtype=torch.float64, device="cuda")
    nk, nb = eps.numel() // eps.shape[-1], eps.shape[-1]
    args = (s, _lib.HF_C128 if eps.dtype == torch.float64 else _lib.HF_C64, method, nk, 1, nb, eps.data_ptr(),
            w.data_ptr(), ne, T, maxiter, _lib.ptr(m0))
    _lib.check(L.hf_find_mu(*args, out.data_ptr()))
    _lib.check(L.hf_find_mu_ws(*args, out[1:].data_ptr(), ws.data_ptr(), ws.numel()))
    return out.tolist()


@pytest.mark.parametrize("nk,nb", [(24577, 8), (160 * 161, 8), (97 * 97, 24), (163841, 1), (40001, 5)])
@pytest.mark.parametrize("T", [0.2, 0.01, 1e-4])
def test_grid_wide_newton_has_the_bits_of_the_cluster_kernel(cuda, nk, nb, T):
    """Method 2 from the threshold of the passes on: the same sums in the same order, so the same bits,
    for starts inside and outside the bracket and for iteration limits that stop in and behind the passes."""
    rng = np.random.default_rng(nk)
    eps = torch.as_tensor(rng.normal(size=(nk, nb)), device="cuda")
    w = rng.uniform(0.5, 1.5, size=nk)
    w = torch.as_tensor(w / w.sum(), device="cuda")
    for ne, mu0, maxiter in ((0.4 * nb, 0.0, 25), (0.4 * nb, -0.2, 25), (0.7 * nb, 40.0, 25), (0.02 * nb, -900.0, 25),
                             (0.4 * nb, 0.3, 1), (0.4 * nb, 0.3, 3), (0.4 * nb, 0.3, 6), (0.4 * nb, 0.3, 8)):
        a, b = _mu_pair(eps, w, ne, T, 2, mu0, maxiter)
        assert a == b, (ne, mu0, maxiter)


@pytest.mark.parametrize("n", [16384, 40000, 131071, 131072, 196612])
@pytest.mark.parametrize("kind,T", [("metal", 0.05), ("gap", 0.01), ("gap", 1e-5), ("staircase", 1e-5), ("flat band", 1e-3),
                                    ("two bands", 0.01), ("narrow", 1e-3), ("single", 0.02)])
def test_certified_bisection_has_the_bits_of_every_level(cuda, n, kind, T):
    """Without a hint, on both sides of the thresholds: in and beside gaps, at temperatures below the spacing of the
    levels, for flat and narrow bands, in single precision, with a short iteration limit."""
    rng = np.random.default_rng(n)
    e = rng.normal(size=(n // 4, 4))
    if kind == "gap":
        e = np.abs(e) + 1.0
        e[:, :2] *= -1.0
    elif kind == "flat band":
        e[:, :2] *= 1e-3
    elif kind == "two bands":
        e = rng.uniform(-1, 1, size=e.shape) - np.where(np.arange(4) < 1, 30.0, 0.0)
    elif kind == "narrow":
        e = 50.0 + 0.01 * e
    dt = torch.float32 if kind == "single" else torch.float64
    eps = torch.as_tensor(e, device="cuda", dtype=dt)
    w = torch.full((n // 4,), 4.0 / n, device="cuda", dtype=dt)
    for ne, maxiter in ((2.0, 0), (0.7, 0), (1.0, 0), (3.37, 0), (0.001, 0), (2.5, 7)):
        a, b = _mu_pair(eps, w, ne, T, 0, None, maxiter)
        assert a == b, (ne, maxiter)


@pytest.mark.parametrize("dt", [np.complex128, np.complex64])
@pytest.mark.parametrize("nk", [1, 257, 400000])
def test_eigh_of_one_band(cuda, dt, nk):
    """nb = 1: the real part (of i A for the Cayley spectral form) and the eigenvector 1, exactly."""
    from jax_hf_b200 import linalg as L
    rng = np.random.default_rng(nk)
    A = (rng.normal(size=(nk, 1, 1)) + 1j * rng.normal(size=(nk, 1, 1))).astype(dt)
    t = torch.as_tensor(A, device="cuda")
    w, V = L.eigh(t)
    assert np.array_equal(w.cpu().numpy()[:, 0], A[:, 0, 0].real) and bool((V == 1).all())
    V1, lam = L.cayley_spectral_setup(t)
    assert np.array_equal(lam.cpu().numpy()[:, 0], -A[:, 0, 0].imag) and bool((V1 == 1).all())


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_certified_bisection_with_a_non_finite_eigenvalue(cuda, bad):
    """A non-finite eigenvalue below the threshold of the grid-wide passes: no bracket, the bits of every level."""
    rng = np.random.default_rng(6)
    e = rng.normal(size=(9000, 3))
    e[77, 1] = bad
    w = torch.full((9000,), 1.0 / 9000, dtype=torch.float64, device="cuda")
    a, b = _mu_pair(torch.as_tensor(e, device="cuda"), w, 1.1, 0.05, 0, None)
    assert a == b or (a != a and b != b)
