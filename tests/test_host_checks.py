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
