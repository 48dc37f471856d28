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
