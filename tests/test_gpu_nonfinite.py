"""A geometry that has run away (a NaN coordinate) gives NaN integrals, matrices
and gradients, as the formulas do, and reads nothing outside the tables."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pyquante_b200 import Ints, _lib, geometries  # noqa: E402
from pyquante_b200.Basis.basis import BasisSet  # noqa: E402
from pyquante_b200.engine import BasisEngine  # noqa: E402
from pyquante_b200.force import rhf_gradient_from_density  # noqa: E402


@pytest.fixture
def lost():
    """Water / 6-31G* whose last hydrogen has a NaN coordinate: (molecule,
    basis, whether each function is that hydrogen's)."""
    mol = geometries.water()
    x, y, z = mol.atoms[2].r
    mol.atoms[2].update_coords([x, float("nan"), z])
    bs = BasisSet(mol, "6-31g*")
    return mol, bs, np.array([bf.atid == mol.atoms[2].atid for bf in bs.bfs])


def test_one_electron_integrals(lost):
    mol, bs, gone = lost
    S, h = Ints.get1ints(bs, mol)
    whole = geometries.water()
    S0, _ = Ints.get1ints(BasisSet(whole, "6-31g*"), whole)
    kept = ~gone[:, None] & ~gone[None, :]
    assert np.array_equal(S[kept], S0[kept]) and np.isnan(S[~kept]).all()
    assert np.isnan(h).all()   # every element sees the lost nucleus


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
def test_two_electron_matrices_and_gradient(lost, mode):
    mol, bs, _ = lost
    eng = BasisEngine(bs.bfs)
    D = torch.eye(eng.nbf, dtype=torch.float64, device=eng.device) + 0.1
    for _ in range(2):   # launched, then replayed
        J, K = eng.jk(D, mode)
        assert bool(J.isnan().all()) and bool(K.isnan().all())
    g = rhf_gradient_from_density(mol, eng, D, D, precision=mode)
    assert np.isnan(g).all()
    assert bool(eng.eri_packed().isnan().any())


def test_coulomb_matrix_in_the_hermite_basis(lost):
    """The Hermite lists are sorted and cut by the Schwarz factors, which are
    NaN here: the quartets that the plan keeps must not be lost."""
    _, bs, _ = lost
    eng = BasisEngine(bs.bfs)
    eng.ctx.check(eng.ctx.lib.pqb_set_param(eng.ctx.h, _lib.PQB_PARAM_HERMITE, 0, 0))   # at any size
    D = torch.eye(eng.nbf, dtype=torch.float64, device=eng.device) + 0.1
    assert np.isnan(eng.schwarz()).any()
    for _ in range(3):
        assert bool(eng.j(D).isnan().all())
