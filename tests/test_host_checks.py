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
    """hf_eigh_warm has no dtype argument and takes 16-byte elements."""
    with pytest.raises(TypeError, match="complex128"):
        linalg.eigh_jacobi(torch.zeros((3, 4, 4), dtype=dtype))


def test_eigh_jacobi_refuses_more_bands_than_the_kernel(no_library):
    with pytest.raises(ValueError, match="nb"):
        linalg.eigh_jacobi(torch.zeros((3, 9, 9), dtype=torch.complex128))


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
