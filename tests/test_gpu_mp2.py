"""GPU parity of the AO -> MO transformation and MP2 (PyQuante/MP.py:20-97)
through the C ABI gather kernels and FP64 GEMMs, against the oracle's
restatement (oracle/pyq_oracle.py: the reference's loops and a dense numpy
transform) and the reference's own MP2 known answers.

Tolerances: 1e-10 on MO integrals and MP2 energies against the oracle on
the same orbitals; the reference's test tolerances on total energies."""
import numpy as np
import pytest

import pyq_oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pyquante_b200 import MP, Ints, _lib, geometries  # noqa: E402
from pyquante_b200.Basis.basis import BasisSet  # noqa: E402
from pyquante_b200.hartree_fock import rhf  # noqa: E402
from pyquante_b200.Molecule import Molecule  # noqa: E402

TOL = 1e-10
SCF = dict(ConvCriteria=1e-12, MaxIter=200, DoAveraging=True)


def oracle_bfs(bs):
    return [O.BF(bf.origin, bf.powers, list(zip(bf.pexps, bf.pcoefs))) for bf in bs.bfs]


def _scf(mol, basis):
    bs = BasisSet(mol, basis)
    S, h, ints = Ints.getints(bs, mol)
    e, orbe, orbs = rhf(mol, bfs=bs, integrals=(S, h, ints), **SCF)
    return bs, ints, e, orbe, orbs


def test_transform_packed_mo_integrals_vs_reference_loops():
    """Water / STO-3G: every slot of the packed MO array equals the
    step-by-step TransformIntsMP2 of the reference on the same orbitals."""
    mol = geometries.water()
    bs, ints, _, orbe, orbs = _scf(mol, "sto-3g")
    mo = MP.TransformIntsMP2(ints, orbs, 5)
    ref = O.transform_ints_mp2_loops(ints.numpy(), orbs, 5)
    assert len(mo) == len(ref)
    assert np.abs(mo.numpy() - ref).max() < TOL


def test_transform_and_mp2_vs_dense_oracle_two_waters():
    """(H2O)2 / 6-31G** (N = 50): MO integrals (ai|bj) and the MP2 energy
    against the dense numpy transform of the oracle's integrals, on the GPU
    SCF's orbitals."""
    mol = geometries.water_cluster(2, seed=4)
    bs, ints, _, orbe, orbs = _scf(mol, "6-31g**")
    n, nocc = len(bs), mol.get_nel() // 2
    orc = O.orc_get2ints(oracle_bfs(bs))
    Z = O.transform_ovov(orc, orbs, nocc)
    mo = MP.TransformIntsMP2(ints, orbs, nocc).numpy()
    k = np.array([O.ijkl2intindex(a, i, b, j) for a in range(nocc) for i in range(0, n, 7) for b in range(nocc)
                  for j in range(0, n, 5)])
    want = np.array([Z[a, i, b, j] for a in range(nocc) for i in range(0, n, 7) for b in range(nocc)
                     for j in range(0, n, 5)])
    assert np.abs(mo[k] - want).max() < TOL
    emp2 = MP.MP2(ints, orbs, orbe, nocc, n - nocc)
    eo = O.mp2(orc, orbs, orbe, nocc, n - nocc)
    print("(H2O)2 MP2 %.12f oracle %.12f" % (emp2, eo))
    assert abs(emp2 - eo) < TOL


def test_mp2_reference_test_energies():
    """The reference's MP2 tests: Tests/h2_mp2.py (1e-6), Tests/he_mp2.py
    (1e-4), Tests/lih_mp2.py and Tests/ch4_mp2.py (GAMESS-UK total and
    correction, 1e-7), all 6-31G**."""
    a2b = 1 / 0.529177249
    cases = [
        (Molecule("h2", [(1, (1.0, 0.0, 0.0)), (1, (-1.0, 0.0, 0.0))]), -1.11591861694, 1e-6, None),
        (Molecule("He", [(2, (0.0, 0.0, 0.0))]), -2.880637, 1e-4, None),
        (Molecule("lih", [(3, (0.0, 0.0, 0.0)), (1, (0.0, 0.0, 1.629912 * a2b))]), -8.0021911, 1e-6, None),
        (Molecule("ch4", [(6, (0, 0, 0)), (1, (0, 0, 1.0836058890)), (1, (1.0216334297, 0, -.3612019630)),
                          (1, (-.5108167148, .8847605034, -.3612019630)),
                          (1, (-.5108167148, -.8847605034, -.3612019630))], units="Angstrom"),
         -40.36985496, 1e-7, -0.16815019),
    ]
    for mol, ref, tol, corr in cases:
        bs, ints, e, orbe, orbs = _scf(mol, "6-31g**")
        nocc = mol.get_nel() // 2
        emp2 = MP.MP2(ints, orbs, orbe, nocc, len(bs) - nocc)
        assert abs(e + emp2 - ref) < tol, (mol.name, e + emp2, ref)
        if corr is not None:
            assert abs(emp2 - corr) < 1e-7


def test_mp2_h2o8_properties():
    """(H2O)8 / 6-31G** (N = 200, 1.6 GB of packed AO integrals, 40 occupied
    orbitals): the correlation energy is negative and does not depend on
    the batching of the first half-transformation."""
    mol = geometries.water_cluster(8, seed=0)
    bs, ints, e, orbe, orbs = _scf(mol, "6-31g**")
    nocc = mol.get_nel() // 2
    e1 = MP.MP2(ints, orbs, orbe, nocc, len(bs) - nocc)
    saved = MP._ROW_BATCH_BYTES
    try:
        MP._ROW_BATCH_BYTES = 37 << 20
        e2 = MP.MP2(ints, orbs, orbe, nocc, len(bs) - nocc)
    finally:
        MP._ROW_BATCH_BYTES = saved
    print("(H2O)8 RHF %.10f MP2 correction %.10f" % (e, e1))
    assert e1 < 0.0 and abs(e1 - e2) < 1e-11


@pytest.mark.parametrize("n,row0,nrows", [(1, 0, 1), (31, 0, 496), (32, 5, 6), (33, 557, 4), (65, 7, 13)])
def test_unpack_rows_at_tile_edges(n, row0, nrows):
    """Copies: equal to the packed array's own elements."""
    P = n * (n + 1) // 2
    ints = torch.arange(P * (P + 1) // 2, dtype=torch.float64, device="cuda")
    out = torch.full((nrows, n, n), -1.0, dtype=torch.float64, device="cuda")
    assert _lib.load().pqb_mo_unpack_rows(_lib.ptr(ints), ints.numel(), n, row0, nrows, _lib.ptr(out),
                                          _lib.stream_ptr()) == _lib.PQB_OK
    k, l = np.indices((n, n))
    KL = np.maximum(k, l) * (np.maximum(k, l) + 1) // 2 + np.minimum(k, l)
    for r in range(nrows):
        hi, lo = np.maximum(KL, row0 + r), np.minimum(KL, row0 + r)
        assert np.array_equal(out[r].cpu().numpy(), hi * (hi + 1) // 2 + lo)


@pytest.mark.parametrize("n,nb,nj,na", [(1, 1, 1, 1), (16, 1, 64, 8), (17, 3, 43, 9), (33, 2, 31, 64), (47, 5, 26, 65),
                                        (30, 7, 11, 130)])
def test_contract_pairs_at_tile_edges(n, nb, nj, na):
    """Against the dense FP64 product: sums of n terms of order one (1e-13
    leaves a hundred roundings)."""
    g = torch.Generator().manual_seed(n)
    P = n * (n + 1) // 2
    Y = torch.randn(nb, P, nj, generator=g, dtype=torch.float64).cuda()
    C = torch.randn(n, na, generator=g, dtype=torch.float64).cuda()
    out = torch.empty(na, n, nb, nj, dtype=torch.float64, device="cuda")
    assert _lib.load().pqb_mo_contract_pairs(_lib.ptr(Y), n, nb, nj, _lib.ptr(C), na, _lib.ptr(out),
                                             _lib.stream_ptr()) == _lib.PQB_OK
    i, j = torch.tril_indices(n, n, device="cuda")
    full = torch.empty(nb, n, n, nj, dtype=torch.float64, device="cuda")
    full[:, i, j] = Y
    full[:, j, i] = Y
    want = torch.einsum("ma,bmnj->anbj", C, full)
    assert float((out - want).abs().max()) < 1e-13 * n * float(want.abs().max().clamp(min=1.0))


@pytest.mark.parametrize("n,nb,row0,nrows", [(1, 1, 0, 1), (7, 3, 2, 26), (8, 8, 0, 36), (9, 9, 44, 1), (25, 17, 3, 300),
                                             (41, 16, 0, 861), (64, 70, 2000, 80), (150, 30, 11000, 325),
                                             (199, 40, 19800, 100), (255, 1, 30000, 20), (289, 18, 41898, 7)])
def test_contract_rows_at_tile_edges(n, nb, row0, nrows):
    """Against the dense FP64 product of the unpacked rows: sums of n terms of
    order one (1e-13 leaves a hundred roundings)."""
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    P = n * (n + 1) // 2
    ints = torch.randn(P * (P + 1) // 2, generator=g, dtype=torch.float64, device="cuda")
    C = torch.randn(n, nb, generator=g, dtype=torch.float64, device="cuda")
    out = torch.full((nb, nrows, n), float("nan"), dtype=torch.float64, device="cuda")
    assert lib.pqb_mo_contract_rows(_lib.ptr(ints), ints.numel(), n, row0, nrows, _lib.ptr(C), nb, _lib.ptr(out),
                                    _lib.stream_ptr()) == _lib.PQB_OK
    X = torch.empty(nrows, n, n, dtype=torch.float64, device="cuda")
    assert lib.pqb_mo_unpack_rows(_lib.ptr(ints), ints.numel(), n, row0, nrows, _lib.ptr(X),
                                  _lib.stream_ptr()) == _lib.PQB_OK
    want = torch.einsum("kb,rkl->brl", C, X)
    assert float((out - want).abs().max()) < 1e-13 * n * float(want.abs().max().clamp(min=1.0))


def _dense_rows(ints, n, row0, nrows):
    """(IJ|kl) of some packed rows as (nrows, n, n), by plain indexing."""
    k, l = torch.meshgrid(torch.arange(n, device="cuda"), torch.arange(n, device="cuda"), indexing="ij")
    KL = torch.maximum(k, l) * (torch.maximum(k, l) + 1) // 2 + torch.minimum(k, l)
    IJ = row0 + torch.arange(nrows, device="cuda")[:, None, None]
    hi, lo = torch.maximum(KL[None], IJ), torch.minimum(KL[None], IJ)
    return ints[hi * (hi + 1) // 2 + lo]


@pytest.mark.parametrize("n,nb", [
    # one of every (strips a warp, warps along l) that a basis of up to 300 functions can get
    (3, 30), (9, 30), (19, 3), (11, 33), (21, 30), (35, 3), (19, 33), (37, 30), (67, 3), (27, 40), (51, 65), (97, 40),
    (35, 33), (67, 65), (129, 40), (43, 40), (85, 30), (161, 40), (51, 40), (99, 65), (193, 40), (59, 40), (117, 30),
    (225, 40), (67, 40), (131, 65), (287, 7), (75, 40), (149, 30)])
def test_contract_rows_in_every_layout(n, nb):
    """Against the dense FP64 product of rows by plain indexing: each of the two
    sums of n terms is off by at most n 2^-53 of the sum of magnitudes."""
    P = n * (n + 1) // 2
    nrows = min(9, P)
    row0 = max(0, P // 2 - 4)   # numbers of the row itself, and of later rows
    g = torch.Generator(device="cuda").manual_seed(n)
    ints = torch.randn(P * (P + 1) // 2, generator=g, dtype=torch.float64, device="cuda")
    C = torch.randn(n, nb, generator=g, dtype=torch.float64, device="cuda")
    out = torch.full((nb, nrows, n), float("nan"), dtype=torch.float64, device="cuda")
    assert _lib.load().pqb_mo_contract_rows(_lib.ptr(ints), ints.numel(), n, row0, nrows, _lib.ptr(C), nb, _lib.ptr(out),
                                            _lib.stream_ptr()) == _lib.PQB_OK
    X = _dense_rows(ints, n, row0, nrows)
    want = torch.einsum("kb,rkl->brl", C, X)
    size = torch.einsum("kb,rkl->brl", C.abs(), X.abs())
    assert bool(((out - want).abs() <= 2 * n * 2.0 ** -53 * size).all())


@pytest.mark.parametrize("n,ncol", [(1, 1), (5, 3), (33, 7)])
def test_unpack_pairs(n, ncol):
    """Copies: rows stored per packed pair, to both orders."""
    P = n * (n + 1) // 2
    Y = torch.arange(P * ncol, dtype=torch.float64, device="cuda").view(P, ncol)
    out = torch.full((n, n, ncol), -1.0, dtype=torch.float64, device="cuda")
    assert _lib.load().pqb_mo_unpack_pairs(_lib.ptr(Y), n, ncol, _lib.ptr(out), _lib.stream_ptr()) == _lib.PQB_OK
    i, j = torch.tril_indices(n, n, device="cuda")
    assert torch.equal(out[i, j], Y) and torch.equal(out[j, i], Y)
