"""The mixed mode's single-precision lists.  Plans below 9 M surviving primitive
quartets run them in FP64, so these systems are above.  Each test asks that
the FP32 kernels ran, a difference from FP64 above 1e-14 of the largest element
(the atomics' order makes 4e-16; integrals of up to 1e-5 that are off by 1e-7
of themselves make more than 1e-13), and that they stay within 1e-5 x 1e-7 x
sums over the density, as the smaller systems' tests do: 1e-8."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pyquante_b200 import _lib, geometries  # noqa: E402
from pyquante_b200.Basis.basis import BasisSet  # noqa: E402
from pyquante_b200.batch import BatchEngine  # noqa: E402
from pyquante_b200.engine import BasisEngine  # noqa: E402

NOISE, BOUND, SAME = 1e-14, 1e-8, 1e-12


def _density(n, seed):
    C = np.random.default_rng(seed).standard_normal((n, max(1, n // 3))) * 0.3
    return torch.as_tensor(C @ C.T, device="cuda")


@pytest.fixture
def eng():
    """(H2O)8 / 6-31G*, 31 M surviving primitive quartets."""
    return BasisEngine(BasisSet(geometries.water_cluster(8, seed=3), "6-31g*").bfs)


def _single_precision(got, want):
    d, top = float((got - want).abs().max()), float(want.abs().max())
    assert NOISE * top < d < BOUND, (d, top)


def test_one_density(eng):
    D = _density(eng.nbf, 1)
    J, K = (x.clone() for x in eng.jk(D, "fp64"))
    for _ in range(3):   # launched, captured, replayed
        Jm, Km = eng.jk(D, "mixed")
        assert eng.plan_counts["fp32"] > 0
        _single_precision(Jm, J)
        _single_precision(Km, K)


def test_two_densities(eng):
    Da, Db = _density(eng.nbf, 2), 0.7 * _density(eng.nbf, 3)
    want = [x.clone() for D in (Da, Db) for x in eng.jk(D, "fp64")]
    single = [x.clone() for D in (Da, Db) for x in eng.jk(D, "mixed")]
    for _ in range(3):
        for got, w, s in zip(eng.jk2(Da, Db, "mixed"), want, single):
            _single_precision(got, w)
            assert float((got - s).abs().max()) < SAME * float(w.abs().max())   # the same FP32 integrals


def test_coulomb_alone(eng):
    eng.ctx.check(eng.ctx.lib.pqb_set_param(eng.ctx.h, _lib.PQB_PARAM_HERMITE, 0, 2**31 - 1))   # the class kernels
    D = _density(eng.nbf, 4)
    J = eng.jk(D, "fp64")[0].clone()
    for _ in range(3):
        _single_precision(eng.j(D, "mixed"), J)


def test_plan_of_several_host_threads(eng):
    D = _density(eng.nbf, 5)
    J, K = (x.clone() for x in eng.jk(D, "mixed"))
    eng.ctx.check(eng.ctx.lib.pqb_set_param(eng.ctx.h, _lib.PQB_PARAM_THREADS, 0, 3))
    eng._plan_key = None
    for got, want in zip(eng.jk(D, "mixed"), (J, K)):
        assert float((got - want).abs().max()) < SAME * float(want.abs().max())


def test_batch_with_a_mask():
    """Three (H2O)5 / 6-31G**, more than 9 M together, in one basis."""
    mols = [geometries.water_cluster(5, seed=s) for s in (2, 3, 4)]
    beng = BatchEngine([(m, "6-31g**") for m in mols])
    counts = beng.plan()
    assert counts["fp32"] > 0
    Ds = [_density(n, 6 + i) for i, n in enumerate(beng.n)]
    flat = torch.cat([d.reshape(-1) for d in Ds])
    J, K = torch.zeros_like(flat), torch.zeros_like(flat)
    for masked in (None, 1):
        mask = None if masked is None else torch.tensor([int(i != masked) for i in range(3)], dtype=torch.int32, device="cuda")
        beng.set_mask(mask)
        beng.jk(flat, J, K, "mixed")
        for i, (m, n, off) in enumerate(zip(mols, beng.n, beng.block_off)):
            blocks = [x[off:off + n * n].view(n, n) for x in (J, K)]
            if i == masked:
                assert not any(bool(b.any()) for b in blocks)
                continue
            want = BasisEngine(BasisSet(m, "6-31g**").bfs).jk(Ds[i], "fp64")
            for b, w in zip(blocks, want):
                _single_precision(b, w)
    beng.set_mask(None)
