"""Calls that go on when an allocation that only serves speed fails.  The failure
is an error code from a stand-in for the allocating runtime call, preloaded
into a child process (nothing is exhausted); it also counts the calls."""
import json
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

FAKE = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int fake_fail_host, fake_fail_device, fake_host, fake_device, fake_launches, fake_graphs;
static void *real(const char *name)
{
    void *h = dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD);
    return h ? dlsym(h, name) : NULL;
}
int cudaHostAlloc(void **p, size_t n, unsigned flags)
{
    ++fake_host;
    return fake_fail_host ? 2 : ((int (*)(void **, size_t, unsigned))real("cudaHostAlloc"))(p, n, flags);
}
int cudaMalloc(void **p, size_t n)
{
    ++fake_device;
    return fake_fail_device ? 2 : ((int (*)(void **, size_t))real("cudaMalloc"))(p, n);
}
int cudaGraphLaunch(void *g, void *s)
{
    ++fake_launches;
    return ((int (*)(void *, void *))real("cudaGraphLaunch"))(g, s);
}
int cudaGraphInstantiate(void **e, void *g, unsigned long long flags)
{
    ++fake_graphs;
    return ((int (*)(void **, void *, unsigned long long))real("cudaGraphInstantiate"))(e, g, flags);
}
"""

PRELUDE = r"""
import ctypes, json, sys
sys.path.insert(0, %r)
import numpy as np
import torch
from pyquante_b200 import Ints, _lib, geometries
from pyquante_b200.Basis.basis import BasisSet
from pyquante_b200.engine import BasisEngine
fake = ctypes.CDLL(None)
class Fake:
    def __getattr__(self, name):
        return ctypes.c_int.in_dll(fake, "fake_" + name).value
    def __setattr__(self, name, value):
        ctypes.c_int.in_dll(fake, "fake_" + name).value = value
f = Fake()
out = {}
""" % ROOT


def _child(tmp_path, program):
    src, lib = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", str(src), "-o", str(lib), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", PRELUDE + program + "\nprint('OUT' + json.dumps(out))"],
                       env=dict(os.environ, LD_PRELOAD=str(lib)), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.rsplit("OUT", 1)[1])


def test_get2jmk_without_page_locked_memory(tmp_path):
    """Repeated calls on numpy arrays go through page-locked copies; without
    them they give the same G by plain copies, and ask for them once."""
    out = _child(tmp_path, r"""
bs = BasisSet(geometries.water(), "sto-3g")
ints = Ints.get2ints(bs, direct=True)
D = np.eye(len(bs)) + 0.1
want = Ints.get2JmK(ints, D)
f.fail_host = 1
before = f.host
out["diff"] = max(float(abs(Ints.get2JmK(ints, D) - want).max()) for _ in range(4))
out["asked"] = f.host - before
""")
    assert out["diff"] < 1e-12 and out["asked"] == 1


HERMITE = r"""
eng = BasisEngine(BasisSet(geometries.water_cluster(2, seed=5), "6-31g**").bfs)
eng.ctx.check(eng.ctx.lib.pqb_set_param(eng.ctx.h, _lib.PQB_PARAM_HERMITE, 0, 0))   # at any size
D = torch.eye(eng.nbf, dtype=torch.float64, device="cuda") + 0.1
for _ in range(3):
    J, K = eng.jk(D)
J0 = torch.empty_like(J)
def j():
    J0.fill_(-1.0)
    eng.j(D, J=J0)
    return float((J0 - J).abs().max())
"""


def test_first_coulomb_build_leaves_the_other_graphs(tmp_path):
    """Making the Hermite lists must not throw away the J/K build's graph."""
    out = _child(tmp_path, HERMITE + r"""
out["diff"] = j()
graphs, launches = f.graphs, f.launches
eng.jk(D, J=J, K=K)
out["graphs"], out["launches"] = f.graphs - graphs, f.launches - launches
""")
    assert out["diff"] < 1e-11 and out["graphs"] == 0 and out["launches"] == 1


def test_coulomb_builds_without_memory_for_the_lists(tmp_path):
    """Without memory for the Hermite lists the class kernels build J, replay
    their graph, leave the J/K graph alone and do not try for the lists at
    every call; the next plan does."""
    out = _child(tmp_path, HERMITE + r"""
f.fail_device = 1
tried = f.device
diffs = [j()]
out["first"] = f.device - tried
tried, launches = f.device, f.launches
diffs += [j() for _ in range(3)]
out["again"], out["replayed"] = f.device - tried, f.launches - launches
graphs = f.graphs
eng.jk(D, J=J, K=K)
out["graphs"] = f.graphs - graphs
f.fail_device = 0
tried = f.device
eng._plan_key = None
diffs += [j() for _ in range(3)]
out["after"] = f.device - tried
out["diff"] = max(diffs)
""")
    assert out["diff"] < 1e-11
    assert out["first"] > 0 and out["again"] == 0 and out["replayed"] == 3 and out["graphs"] == 0 and out["after"] > 0
