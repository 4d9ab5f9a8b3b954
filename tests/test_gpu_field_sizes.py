"""The field solve at the edges of its sizes: every length of the register
FFTs (8 to 8192 points on the doubled grid: one to four stages, threads per
line from one to 1024, several lines and one line per block) against the same
convolution by torch.fft in FP64.

Tolerance: an FFT of N points errs by at most about log2(N) rounding units of
its 2-norm per pass, so the two solves of 2^25 doubled points agree within a
few tens of units: 1e-14 in FP64, taken as 1e-12 (the FP64 Green function,
which cancels, is common to both); 1e-6 in the FP32 form.  Runs of a group of
bunches of one grid size take the same kernels with the members in device
memory and equal the solo runs to the order of the moment sums (1e-10)."""
import numpy as np
import pytest

from conftest import load_impz
from test_gpu_cufft import cufft_potential

pytestmark = pytest.mark.gpu

impz = load_impz()
from impz_b200 import beams  # noqa: E402

SIZES = [(4, 4, 4), (8, 4, 8), (4, 8, 16), (16, 16, 16), (8, 32, 32), (64, 8, 64), (32, 16, 128),
         (32, 64, 256), (16, 8, 512), (64, 64, 1024), (4, 16, 2048), (8, 8, 4096)]


@pytest.mark.parametrize("form,tol", [(impz.FORM_FP64, 1e-12), (impz.FORM_FP32CONV, 1e-6)])
@pytest.mark.parametrize("grid", SIZES)
def test_potential_at_every_length(grid, form, tol):
    cfg = beams.fodo_1e5(n=20_011, seed=beams.SEED0 + 91)
    with impz.Bunch(cfg["pts"], cfg["current"], cfg["mass"], cfg["charge"], cfg["freq"],
                    cfg["refptcl"], grid, form=form, track_ids=False) as b:
        _, _, _, msize = b.sc_prepare(1.0, 1.0)
        rho, _ = b.deposit(want_counts=False)
        phi = b.poisson()
    want = cufft_potential(rho, grid, msize)
    assert np.linalg.norm(phi - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("form", [impz.FORM_FP64, impz.FORM_FP32CONV])
@pytest.mark.parametrize("grid", [(4, 8, 16), (16, 16, 16), (8, 8, 4096), (64, 64, 32), (16, 16, 128),
                                  (16, 16, 256)])
def test_group_equals_solo(grid, form):
    def make(k):
        cfg = beams.fodo_1e5(n=3000 + 1111 * k, seed=beams.SEED0 + 92 + k)
        return impz.Bunch(cfg["pts"], cfg["current"], cfg["mass"], cfg["charge"], cfg["freq"],
                          cfg["refptcl"], grid, form=form, track_ids=False)

    lats = [beams.fodo(1, gradient=10.0 + k) for k in range(3)]
    solo = []
    for k in range(3):
        with make(k) as b:
            solo.append(b.run(lats[k])[0])
    bunches = [make(k) for k in range(3)]
    for (recs, _), want in zip(impz.run_batch(bunches, lats), solo):
        scale = np.max(np.abs(want[:, :44]), axis=0)
        assert np.max(np.abs(recs[:, :44] - want[:, :44]) / scale) <= 1e-10
    for b in bunches:
        b.close()


@pytest.mark.parametrize("grid", [(64, 64, 128), (16, 32, 256)])
def test_the_fp32_field_has_no_net_force_of_its_own(grid):
    """The field of a bunch on itself, summed over its charge, is zero but for
    rounding, which differs from bunch to bunch: 2e-9 to 4e-9 of the rms force
    (the potential errs by 1e-7 in 2-norm; the sum over the bunch averages it).
    A gain or a shift of the transforms that depends on the position or the
    harmonic gives every bunch the same force.  The mean over twelve bunches is
    held to 4e-9 along x and y: three standard deviations of the mean of twelve
    at 4.5e-9."""
    nets = []
    for k in range(12):
        cfg = beams.fodo_1e5(n=200_000, seed=beams.SEED0 + 300 + k)
        field = {}
        for form in (impz.FORM_FP64, impz.FORM_FP32CONV):
            with impz.Bunch(cfg["pts"], cfg["current"], cfg["mass"], cfg["charge"], cfg["freq"],
                            cfg["refptcl"], grid, form=form, track_ids=False) as b:
                b.sc_prepare(1.0, 1.0)
                rho, _ = b.deposit(want_counts=False)
                b.poisson(want_phi=False)
                field[form] = np.reshape(b.kick(0.025, want_e=True), (3, -1))
        rho = rho / rho.sum()
        e = field[impz.FORM_FP64]
        nets.append(((field[impz.FORM_FP32CONV] - e) @ rho / np.sqrt(e ** 2 @ rho))[:2])
    mean = np.mean(nets, axis=0)
    print(grid, "net force", mean, "spread", np.std(nets, axis=0))
    assert np.max(np.abs(mean)) <= 4e-9, mean
