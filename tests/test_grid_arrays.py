"""MolecularGrid's arrays on their way to the kernels, which read and write them
by address: whatever a caller has put in their place is either laid out as
the kernels take it or refused.  Host logic: the library is a stand-in that
computes the density on the CPU and takes no address inside a density whose
rows are not two doubles."""
import ctypes

import numpy as np
import pytest
import torch

from pyquante_b200 import MolecularGrid as M
from pyquante_b200 import _lib
from pyquante_b200 import dft as dft_module

NG, N = 11, 3


class _Kernels:
    def __init__(self, gr):
        self.gr = gr

    def pqb_grid_work(self, ng, n):
        return 1

    def pqb_grid_density(self, ng, n, B, D, rho, stride, copies, work, stream):
        d = self.gr.density
        s = d.untyped_storage()
        inside = s.data_ptr() <= rho.value < s.data_ptr() + s.nbytes()
        assert not inside or (d.dtype == torch.float64 and d.stride() == (2, 1)), "address in another layout"

        def array(p, count):
            return np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_double)), (count,))

        b = array(B, ng * n).reshape(ng, n)
        r = ((b @ array(D, n * n).reshape(n, n)) * b).sum(1)
        out = array(rho, stride * (ng - 1) + copies)
        for c in range(copies):
            out[c::stride] = r
        return _lib.PQB_OK

    def pqb_grid_fock(self, ng, n, B, v, F, work, stream):
        assert self.gr.bfgrid.dtype == torch.float64 and self.gr.bfgrid.shape == (ng, n)

        def array(p, count):
            return np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_double)), (count,))

        b = array(B, ng * n).reshape(ng, n)
        array(F, n * n)[:] = (b.T @ (array(v, ng)[:, None] * b)).ravel()
        return _lib.PQB_OK


@pytest.fixture
def grid(monkeypatch):
    gr = object.__new__(M.MolecularGrid)
    gr.ng, gr.nbf, gr.device = NG, N, torch.device("cpu")
    gr.bfgrid = torch.randn(NG, N, dtype=torch.float64, generator=torch.Generator().manual_seed(1))
    gr.density = torch.zeros(NG, 2, dtype=torch.float64)
    monkeypatch.setattr(M._lib, "load", lambda: _Kernels(gr))
    monkeypatch.setattr(M, "stream_ptr", lambda *a: None)
    return gr


@pytest.mark.parametrize("layout", ["rows", "columns", "strided", "float32"])
@pytest.mark.parametrize("two", [False, True])
def test_any_layout_of_the_density_is_filled(grid, layout, two):
    if layout == "columns":
        grid.density = torch.zeros(2, NG, dtype=torch.float64).T
    elif layout == "strided":
        grid.density = torch.zeros(NG, 4, dtype=torch.float64)[:, ::2]
    elif layout == "float32":
        grid.density = torch.zeros(NG, 2, dtype=torch.float32)
    rho = grid.density
    D = np.arange(9.0).reshape(3, 3)
    grid.set_density(D, 2.0 * D if two else None)
    want = ((grid.bfgrid @ torch.as_tensor(D)) * grid.bfgrid).sum(1)
    assert grid.density is rho
    tol = 1e-5 if layout == "float32" else 1e-12
    assert torch.allclose(rho[:, 0].double(), want, rtol=tol, atol=tol)
    assert torch.allclose(rho[:, 1].double(), 2.0 * want if two else want, rtol=tol, atol=tol)


def test_amplitudes_and_values_of_another_type_are_refused(grid):
    D, v = np.eye(N), torch.ones(NG, dtype=torch.float64)
    for bad in (torch.ones(NG), torch.ones(NG - 1, dtype=torch.float64),
                torch.ones(NG, dtype=torch.float64, device="meta")):
        with pytest.raises(RuntimeError):
            grid.fock(bad)
    good = grid.bfgrid
    for bad in (good.float(), good[:-1], good.to("meta")):
        grid.bfgrid = bad
        with pytest.raises(RuntimeError):
            grid.set_density(D)
        with pytest.raises(RuntimeError):
            grid.fock(v)


def test_fock_of_amplitudes_that_a_caller_has_set(grid):
    """getXC's matrix needs amplitudes and no basis: a caller may bring them."""
    grid.nbf = 0
    v = torch.linspace(-1.0, 1.0, NG, dtype=torch.float64)
    want = grid.bfgrid.T @ (v[:, None] * grid.bfgrid)
    assert torch.allclose(grid.fock(v), want, rtol=1e-12, atol=1e-12)


def _xc_stub(rho, gamma, functional):
    return (rho.sum(0), rho[0].contiguous(), rho[1].contiguous(), None, None, None)


def test_getxc_of_a_zero_density_raises_and_leaves_it(grid, monkeypatch):
    monkeypatch.setattr(dft_module, "XC", _xc_stub)
    grid.xyzw = torch.ones(NG, 4, dtype=torch.float64)
    grid.density = torch.full((NG, 2), 1e-12, dtype=torch.float64)   # below the floor
    with pytest.raises(ZeroDivisionError):
        dft_module.getXC(grid, 10)
    assert torch.equal(grid.density, torch.zeros(NG, 2, dtype=torch.float64))
    grid.density = torch.full((NG, 2), 0.25, dtype=torch.float64)
    exc, F = dft_module.getXC(grid, 10)
    assert abs(float(grid.density.sum()) - 10.0) < 1e-12 and abs(exc - 10.0) < 1e-12
