"""What the host enqueues, without a GPU: the library's objects linked with a
recording CUDA runtime (fake_cudart.cpp; kernels do not run).

A packed advance whose k-th enqueued operation fails, for every k, returns the
error and frees its argument memory only after everything it had enqueued, on
both streams.

impz_kernel_launches counts the kernels that ran: in every call that launches
any, by direct launches and by graph replay alike.

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


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_the_launch_count_is_the_number_of_kernels(fake_lib, form):
    run_child(fake_lib, "launch_counts_" + form)


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


def launch_counts(form):
    impz, L, beams = setup()
    from test_wake import synthetic_table

    def counted(what, f, want=None):
        c0, k0 = impz.kernel_launches(), L.fake_kernels()
        f()
        c, k = impz.kernel_launches() - c0, L.fake_kernels() - k0
        assert c == k, (what, c, k)
        assert want is None or c == want, (what, c, want)

    drift = impz.elem(0, 0.1, 4, 1, [1.0])
    for grid in ((8, 8, 16), (64, 16, 8)):
        b = make(impz, beams, 700, grid, form)
        counted("map", lambda: b.map_half(drift, 0.0, 0.0, 0.0125, 1, 0), 1)
        counted("prepare", lambda: b.sc_prepare(1.0, 1.0))
        counted("deposit", lambda: b.deposit(), 3)
        counted("poisson", lambda: b.poisson())
        counted("kick", lambda: b.kick(0.025, want_e=True))
        counted("moments", lambda: b.moments())
        counted("bunching", lambda: b.bunching(1e3))
        # a prologue, then ten kernels a step: in pairs from a graph, and singly
        counted("capture", lambda: b.run([drift]), 1 + 4 * 10)
        counted("replay", lambda: b.run([drift]), 1 + 4 * 10)
        counted("odd", lambda: b.run([impz.elem(0, 0.1, 3, 1, [1.0])]), 1 + 3 * 10)
        b.wake(synthetic_table(), 1.0, True)
        counted("wake", lambda: b.run([drift]), 1 + 4 * 12)
        b.wake_off()
        b.profile_enable(True)
        counted("profile", lambda: b.run([drift]), 1 + 4 * 10)
        b.profile_enable(False)
        c = beams.fodo_1e5(n=700)
        counted("upload", lambda: b.upload(c["pts"], c["current"], c["refptcl"]))
        counted("download", lambda: b.download())
        b.close()
    # groups: the field solve once per grid size, the rest once
    grids = [(8, 8, 16), (16, 8, 16), (8, 8, 16)]
    for group, per in (((0, 2), 10), ((0, 1, 2), 17)):
        bs = [make(impz, beams, 500, grids[k], form) for k in group]
        lats = [[drift]] * len(bs)
        for _ in range(2):
            counted("batch", lambda: impz.run_batch(bs, lats), len(bs) + 4 * per)
            counted("packed", lambda: impz.run_packed(bs, lats, 3), len(bs) + 4 * per)
        for b in bs:
            b.close()
    # the deposit into the caller's memory (host memory here)
    x = [np.zeros(64) for _ in range(6)]
    box = np.array([-1.0, 1.0] * 3)
    out = np.zeros(8 * 8 * 8)
    for n, want in ((64, 3), (0, 2)):
        counted("static", lambda: L.impz_deposit_static(
            *[a.ctypes.data for a in x], n, 2.0, 1.0, 1.0, 4e8, 1.0,
            box.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), 8, 8, 8, out.ctypes.data, None),
            want)


if __name__ == "__main__":
    if sys.argv[1] == "packed_failures":
        packed_failures()
    else:
        form = load_impz().FORM_FP64 if sys.argv[1].endswith("64") else load_impz().FORM_FP32CONV
        launch_counts(form)
