"""One-electron kernels at the edges of their splits: s to f functions, one
primitive pair to more than a warp's 32, one atom to more than a warp's lanes
and more than the gradient's shared sums hold."""
import ctypes

import numpy as np
import pytest

import pyq_oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pyquante_b200 import _lib  # noqa: E402
from pyquante_b200.CGBF import CGBF  # noqa: E402
from pyquante_b200.engine import FunctionTable, oneint  # noqa: E402

POWERS = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (2, 0, 0), (0, 1, 1), (0, 0, 3), (1, 1, 1), (0, 2, 1)]


class _Nucleus:
    def __init__(self, z, r):
        self.atno, self.r = z, r

    def pos(self):
        return tuple(self.r)


def _system(natoms, nfun, nprim, seed):
    rng = np.random.default_rng(seed)
    nuclei = [_Nucleus(int(rng.integers(1, 10)), rng.uniform(-3.0, 3.0, 3)) for _ in range(natoms)]
    bfs = []
    for f in range(nfun):
        bf = CGBF(nuclei[f % natoms].pos(), POWERS[f % len(POWERS)], f % natoms)
        for _ in range(nprim):
            bf.add_primitive(float(np.exp(rng.uniform(np.log(0.15), np.log(300.0)))), float(rng.uniform(0.1, 0.6)))
        bfs.append(bf)
    return bfs, nuclei


@pytest.mark.parametrize("natoms,nfun,nprim", [(1, 1, 1), (3, 8, 6), (31, 9, 2), (33, 5, 1), (300, 4, 2)])
def test_oneint_matches_the_oracle(natoms, nfun, nprim):
    bfs, nuclei = _system(natoms, nfun, nprim, seed=natoms)
    S, T, V = (x.cpu().numpy() for x in oneint(FunctionTable(bfs, 0), nuclei, _lib.context(0)))
    obfs = [O.BF(bf.origin, bf.powers, list(zip(bf.pexps, bf.pcoefs))) for bf in bfs]
    So, ho = O.orc_get1ints(obfs, [(a.atno, tuple(a.r)) for a in nuclei])
    # the primitives' own scale: a few hundred FP64 roundings of sums of |terms|
    assert np.abs(S - So).max() < 1e-13 * max(1.0, np.abs(So).max())
    assert np.abs(T + V - ho).max() < 1e-12 * max(1.0, np.abs(T).max(), np.abs(V).max())


def _grad(bfs, nuclei, D, W, charges=None):
    n, nat = len(bfs), len(nuclei)
    ctx = _lib.context(0)
    ft = FunctionTable(bfs, 0)
    g = torch.zeros(3 * nat, dtype=torch.float64, device="cuda")
    fa = torch.tensor([bf.atid for bf in bfs], dtype=torch.int32, device="cuda")
    xyz = (ctypes.c_double * (3 * nat))(*[c for a in nuclei for c in a.pos()])
    z = (ctypes.c_double * nat)(*(charges if charges is not None else [float(a.atno) for a in nuclei]))
    Dd, Wd = (torch.as_tensor(x, device="cuda") for x in (D, W))
    assert Dd.shape == (n, n)
    ctx.check(ctx.lib.pqb_grad_1e(ctx.h, *ft.args(), _lib.ptr(fa), nat, xyz, z, _lib.ptr(Dd), _lib.ptr(Wd),
                                  _lib.ptr(g), _lib.stream_ptr()))
    return g.cpu().numpy().reshape(nat, 3)


def _shifted(bf, x, d):
    """The functions 2 alpha g_(l+1x) (d = 1) or l_x g_(l-1x) (d = -1) of a
    contracted function, as (powers, [(exponent, plain coefficient)])."""
    pw = list(bf.powers)
    pw[x] += d
    f = (lambda e: 2.0 * e) if d > 0 else (lambda e: float(bf.powers[x]))
    return tuple(pw), [(e, f(e) * c * m) for e, c, m in zip(bf.pexps, bf.pcoefs, bf.pnorms)]


def _oracle_grad(bfs, nuclei, D, W):
    """The gradient from the oracle's own integrals over raised and lowered
    functions, nucleus by nucleus."""
    n, nat = len(bfs), len(nuclei)
    g = np.zeros((nat, 3))
    plain = [(bf.origin, bf.powers, [(e, c * m) for e, c, m in zip(bf.pexps, bf.pcoefs, bf.pnorms)]) for bf in bfs]
    for x in range(3):
        shifted, sign, of = [], [], []
        for i, bf in enumerate(bfs):
            for d in (1, -1):
                if d < 0 and bf.powers[x] == 0:
                    continue
                pw, prims = _shifted(bf, x, d)
                shifted.append((bf.origin, pw, prims))
                sign.append(d)
                of.append(i)
        # primitives that the oracle would normalise: divide its norm out again
        obfs = []
        for origin, powers, prims in plain + shifted:
            unit = [O.BF(origin, powers, [(e, 1.0)]) for e, _ in prims]
            obfs.append(O.BF(origin, powers, [(e, c / u.pnorms[0]) for (e, c), u in zip(prims, unit)]))
        dS = np.zeros((n, n))
        for c in [None] + list(range(nat)):
            at = [] if c is None else [(nuclei[c].atno, tuple(nuclei[c].r))]
            S, h = O.orc_get1ints(obfs, at)
            if c is None:
                S0, T0 = S, h
            dh = np.zeros((n, n))   # <d chi_i/dA_x | T or V_c | chi_j>
            for r, (s, i) in enumerate(zip(sign, of)):
                dh[i] += s * (h if c is None else h - T0)[n + r, :n]
                if c is None:
                    dS[i] += s * S0[n + r, :n]
            q = 2.0 * (D + D.T) * dh
            if c is None:
                q = q - 2.0 * (W + W.T) * dS
            for i, bf in enumerate(bfs):
                g[bf.atid, x] += q[i].sum()
            if c is not None:
                g[c, x] -= q.sum()
    return g


@pytest.mark.parametrize("natoms,nfun,nprim", [(1, 2, 1), (3, 8, 6), (33, 6, 2)])
def test_gradient_matches_the_oracle(natoms, nfun, nprim):
    """Unsymmetric D and W; a few hundred FP64 roundings of sums of terms that
    reach the kinetic derivative's 2 alpha sqrt(alpha) of the tightest
    primitive (1e4)."""
    bfs, nuclei = _system(natoms, nfun, nprim, seed=50 + natoms)
    rng = np.random.default_rng(natoms)
    D, W = rng.standard_normal((2, nfun, nfun))
    g, go = _grad(bfs, nuclei, D, W), _oracle_grad(bfs, nuclei, D, W)
    assert np.abs(g - go).max() < 1e-9 * max(1.0, np.abs(go).max())


def test_gradient_of_many_nuclei_is_the_sum_of_their_parts():
    """More nuclei than the shared sums hold: linear in the charges, so the
    halves' attraction adds up."""
    bfs, nuclei = _system(300, 5, 2, seed=9)
    rng = np.random.default_rng(1)
    D, W = rng.standard_normal((2, 5, 5))
    z = np.array([float(a.atno) for a in nuclei])
    lo = np.where(np.arange(300) < 150, z, 0.0)
    g, gl, gh, g0 = (_grad(bfs, nuclei, D, W, c) for c in (z, lo, z - lo, 0.0 * z))
    assert np.abs(g - (gl + gh - g0)).max() < 1e-11 * max(1.0, np.abs(g).max())
    few = _grad(bfs, nuclei[:150], D, W, z[:150])
    assert np.abs(gl[:150] - few).max() < 1e-11 * max(1.0, np.abs(few).max())
