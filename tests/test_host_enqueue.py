"""What the host enqueues, without a GPU: the library's objects linked with a
recording CUDA runtime (fake_cudart.cpp; kernels do not run).

A packed advance whose k-th enqueued operation fails, for every k, returns the
error and frees its argument memory only after everything it had enqueued, on
both streams.

The process (a child: the library is loaded a second time) is given the linked
library's path."""
import ctypes
import importlib.util
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, load_impz

CHILD = os.environ.get("IMPZ_FAKE_LIB")


def _build_module():
    spec = importlib.util.spec_from_file_location(
        "impz_build", os.path.join(ROOT, "impact-z_b200", "build.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    b = _build_module()
    b.build_lib()
    out = str(tmp_path_factory.mktemp("fake") / "libimpz_fake.so")
    objs = [os.path.join(b.OBJ, u + ".o") for u in [s for s, _ in b.UNITS] + b.HOST_UNITS]
    cuda = os.path.join(os.path.dirname(os.path.dirname(b.nvcc())), "include")
    b._run([b.host_cxx(), "-shared", "-fPIC", "-O1", "-std=c++17", "-I", cuda, "-o", out,
            os.path.join(ROOT, "tests", "fake_cudart.cpp")] + objs + ["-lpthread"])
    return out


def run_child(fake_lib, what):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), what],
                       env=dict(os.environ, IMPZ_FAKE_LIB=fake_lib), timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_a_failed_packed_advance_frees_its_arguments_after_all_its_work(fake_lib):
    run_child(fake_lib, "packed_failures")


# ---- in the child ---------------------------------------------------------
def setup():
    impz = load_impz()
    impz.LIB_PATH = CHILD
    L = impz.lib()
    for f in ("fake_ops", "fake_kernels", "fake_faults"):
        getattr(L, f).restype = ctypes.c_longlong
    L.fake_fail_at.argtypes = [ctypes.c_longlong]
    from impz_b200 import beams
    return impz, L, beams


def make(impz, beams, n, grid, form):
    c = beams.fodo_1e5(n=n)
    return impz.Bunch(c["pts"], c["current"], c["mass"], c["charge"], c["freq"], c["refptcl"], grid,
                      form=form, track_ids=False)


def packed_failures():
    impz, L, beams = setup()
    lat = beams.fodo(1)

    def advance(fail_at):
        bs = [make(impz, beams, 500 + 100 * k, g, impz.FORM_FP64)
              for k, g in enumerate([(8, 8, 16), (16, 8, 16), (8, 8, 16)])]
        arrs = [impz.elem_array(lat) for _ in bs]
        for b, a in zip(bs, arrs):
            assert L.impz_run_begin(b.h, a, len(lat)) == 0
        hs = (ctypes.c_void_p * len(bs))(*[b.h for b in bs])
        L.fake_fail_at(fail_at)
        rc = L.impz_run_advance_packed(hs, len(bs), 2, None)
        n, faults = L.fake_ops(), L.fake_faults()
        L.fake_fail_at(-1)
        for b in bs:
            b.close()
        return rc, n, faults

    rc, total, faults = advance(10**9)
    assert rc == 0 and faults == 0 and total > 40, (rc, total, faults)
    bad = []
    for k in range(total):
        before = L.fake_faults()
        rc, _, faults = advance(k)
        if rc != impz.ERR_CUDA or faults != before:
            bad.append((k, rc, faults - before))
    assert not bad, "%d of %d: %s" % (len(bad), total, bad)


if __name__ == "__main__":
    {"packed_failures": packed_failures}[sys.argv[1]]()
