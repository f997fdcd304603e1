"""Checks that the Python entry points make before they hand pointers to the library (CPU only)."""

import numpy as np
import pytest
import torch

from jax_hf_b200 import _lib, linalg


class _NoLibrary:
    """Stands in for the library: any call is a failure of the check before it."""

    def __getattr__(self, name):
        raise AssertionError(f"{name} was reached")


@pytest.fixture
def no_library(monkeypatch):
    monkeypatch.setattr(_lib, "lib", lambda: _NoLibrary())
    monkeypatch.setattr(_lib, "stream_ptr", lambda device=None, *a: 0)


@pytest.mark.parametrize("dtype", [torch.complex64, torch.float32, torch.float64])
def test_eigh_jacobi_refuses_other_element_sizes(no_library, dtype):
    """The SCF loop's eigensolver takes 16-byte elements."""
    with pytest.raises(TypeError, match="complex128"):
        linalg.eigh_jacobi(torch.zeros((3, 4, 4), dtype=dtype))


@pytest.mark.parametrize("dtype", [torch.complex64, torch.complex128, torch.float64])
def test_objective_hands_complex128_to_its_node(monkeypatch, dtype):
    """The node's backward passes P and h to kernels that read 16-byte elements."""
    from types import SimpleNamespace

    from jax_hf_b200 import adjoint
    seen = []
    monkeypatch.setattr(adjoint._ObjectiveFn, "apply", staticmethod(lambda *a: seen.append(a)))
    P = torch.zeros((2, 3, 4, 4), dtype=dtype).transpose(-1, -2)
    adjoint.objective(P, torch.zeros(2, 3, 4), SimpleNamespace(dtype=torch.complex128), torch.zeros_like(P))
    P1, p1, h1, _ = seen[0]
    assert P1.dtype == h1.dtype == torch.complex128 and p1.dtype == torch.float64
    assert P1.is_contiguous() and h1.is_contiguous()


def test_cotangents_are_materialised():
    """Autograd passes conj() and negated views without writing their numbers; the kernels read memory."""
    from jax_hf_b200 import adjoint
    x = torch.randn(2, 3, 3, dtype=torch.complex128)
    g = adjoint._cotangent(x.conj())
    assert not g.is_conj() and torch.equal(torch.view_as_real(g), torch.view_as_real(x.conj().resolve_conj()))
    y = torch.randn((), dtype=torch.complex128).conj().imag
    assert y.is_neg()
    z = adjoint._dev_scalar(y, y.device)
    assert not z.is_neg() and float(z) == float(y)


@pytest.mark.parametrize("engine", [0, _lib.FOCK_TILE_PLAN, _lib.FOCK_PIPE, _lib.FOCK_GENERIC_FFT])
@pytest.mark.parametrize("n1,n2,nb", [(340, 24, 5), (340, 24, 9), (430, 24, 3), (120, 120, 8)])
def test_scf_workspace_covers_the_builds_of_the_loop(engine, n1, n2, nb):
    """The SCF driver builds without the two-factor passes, whose slot plan may be the smaller one: its
    workspace is the one of a problem that asks for that itself."""
    import ctypes as C

    from jax_hf_b200.reference_scf import SCFConfig, _scf_config_struct, _ScfConfig
    from jax_hf_b200.solver import _CgProblem
    L = _lib.lib()
    cf = _scf_config_struct(SCFConfig())
    fn = L.hf_scf_workspace_size
    fn.argtypes, fn.restype = [C.POINTER(_CgProblem), C.POINTER(_ScfConfig), C.POINTER(C.c_size_t)], C.c_int
    sizes = []
    for extra in (0, _lib.FOCK_NO_TWO_FACTOR):
        pb = _CgProblem(n1, n2, nb, _lib.FOCK_EXCHANGE | _lib.FOCK_VR_REAL | engine | extra, 0.1, 1.0, 1.0)
        need = C.c_size_t(0)
        _lib.check(fn(C.byref(pb), C.byref(cf), C.byref(need)))
        sizes.append(need.value)
    assert sizes[0] == sizes[1]


def _kernels():
    """(file, name, parameters, body) of every __global__ function in the sources."""
    import re
    from pathlib import Path
    csrc = Path(__file__).resolve().parents[1] / "jax_hf_b200" / "csrc"
    for f in sorted([*csrc.glob("*.cu"), *csrc.glob("*.cuh")]):
        s = f.read_text()
        for m in re.finditer(r"__global__", s):
            head = s[m.start():s.index("{", m.start())]
            if ";" in head:
                continue
            bounds = re.match(r"__global__\s+void\s*(__launch_bounds__\s*\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\))?", head)
            rest = head[bounds.end():]
            depth, i = 1, m.start() + len(head) + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(s[i], 0)
                i += 1
            yield f.name, rest[:rest.index("(")].strip(), rest[rest.index("("):], s[m.start() + len(head):i]


def test_dependently_launched_kernels_read_through_plain_pointers():
    """A kernel launched with programmatic serialization starts while its predecessor still writes what it will
    read and reads what it will write.  __restrict__ would let the compiler read through the non-coherent
    path, and move accesses across the wait: both take memory that no one else touches while the kernel runs."""
    seen, bad = 0, []
    for f, name, params, body in _kernels():
        if "pdl_begin()" in body or "pdl_wait()" in body:
            seen += 1
            if "__restrict__" in params:
                bad.append(f"{f}: {name}")
    assert seen > 30 and not bad, bad
