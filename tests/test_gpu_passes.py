"""Runs whose steps change the instantiation of the particle pass (drifts and
linear maps, other maps, ideal RF gaps), and wakes over few and many planes,
against the oracle at particle counts from a fraction of one warp pair to
several iterations of a block.

Tolerance: FP64 run tolerance, every record's rms columns within 1e-8 of the
oracle, and 1e-5 of the rms sizes, momenta and emittances in the
FP32-convolution form.  A group of runs takes one instantiation for all its
members, so its records equal the solo runs' up to the order of the moment sums
(1e-10); in the FP32 form the instantiations may contract differently, and a
last bit that reaches an FP32 weight or charge is 6e-8 of one particle or node
(1e-9 of a moment)."""
import numpy as np
import pytest

from conftest import load_impz, load_oracle
from test_wake import synthetic_table

pytestmark = pytest.mark.gpu

impz = load_impz()
orc = load_oracle()
from impz_b200 import beams  # noqa: E402

RMS_COLS = [6, 7, 8, 9, 11, 12, 13, 14, 15, 17, 18, 19, 20, 21, 23]
FP32_COLS = [7, 9, 11, 13, 15, 17, 19, 21, 23]  # sizes, momenta, emittances

DRIFT = impz.elem(0, 0.05, 1, 1, [1.0])
BEND = impz.elem(4, 0.05, 1, 1, [0.0125, 0.0, 150.0, 0.01, 0.0, 0.0, 0.0, 0.0, 0.0])
GAP = impz.elem(101, 0.05, 1, 1, [1.0e6, 402.5e6, -30.0, -1.0, 1.0])
# one-step elements, so that steps are launched singly and, at two equal
# neighbours, as a pair; one ends in the middle of such a pair
ORDERS = {"light": [DRIFT] * 5, "maps": [DRIFT, BEND, BEND, DRIFT, DRIFT, BEND],
          "full": [GAP, DRIFT, DRIFT, GAP, GAP, DRIFT],
          "all": [DRIFT, GAP, BEND, BEND, DRIFT, DRIFT, BEND, GAP, GAP, BEND, DRIFT]}


def config(n, grid=(16, 16, 16)):
    cfg = beams.fodo_1e5(n=n, seed=beams.SEED0 + 95)
    cfg["grid"] = grid
    return cfg


def bunch(cfg, form=impz.FORM_FP64, **kw):
    return impz.Bunch(cfg["pts"], cfg["current"], cfg["mass"], cfg["charge"], cfg["freq"],
                      cfg["refptcl"], cfg["grid"], form=form, track_ids=False, **kw)


def compare(b, lattice, cfg, wake=None, cols=RMS_COLS, tol=1e-8):
    try:
        if wake is not None:
            orc.wake_set(*wake)
        want, _, _ = orc.run(lattice, cfg["pts"], cfg["current"], cfg["mass"], cfg["charge"],
                             cfg["freq"], cfg["refptcl"], cfg["grid"])
    finally:
        orc.wake_off()
    recs, zs = b.run(lattice)
    np.testing.assert_allclose(zs, want[:, 0], rtol=0, atol=0)
    refs = b.run_reference()
    got = np.array([impz.diag_row(zs[i], recs[i], refs[i], cfg["mass"], cfg["freq"])
                    for i in range(len(recs))])
    for c in cols:
        scale = np.max(np.abs(want[:, c])) + 1e-300
        assert np.max(np.abs(got[:, c] - want[:, c])) <= tol * scale, c


@pytest.mark.parametrize("order", list(ORDERS))
@pytest.mark.parametrize("n", [33, 20_011])
def test_steps_of_every_pass_match_the_oracle(order, n):
    cfg = config(n)
    with bunch(cfg) as b:
        compare(b, ORDERS[order], cfg)


@pytest.mark.parametrize("order", list(ORDERS))
@pytest.mark.parametrize("n", [33, 20_011])
def test_steps_of_every_pass_in_the_fp32_form(order, n):
    cfg = config(n)
    with bunch(cfg, impz.FORM_FP32CONV) as b:
        compare(b, ORDERS[order], cfg, cols=FP32_COLS, tol=1e-5)


def ions(n):
    half = n // 3
    pts, ref, mass, _ = beams.charge_state_bunch([n - half, half], (33.0, 34.0), [4e-4, 3e-4],
                                                 seed=beams.SEED0 + 97)
    return dict(pts=pts, refptcl=ref, current=7e-4, mass=mass, charge=33.0, freq=80.5e6,
                grid=(16, 16, 16))


@pytest.mark.parametrize("strength", [30.0, -30.0, 0.0, 1e-3, -1e-3])
@pytest.mark.parametrize("form", [impz.FORM_FP64, impz.FORM_FP32CONV])
def test_kmap_quadrupole_of_two_charge_states_per_particle(form, strength):
    """One half map without space charge.  Both forms compute it in FP64: some
    twenty roundings of a column's largest value (1e-13 of its rms); sinh from
    exp(x), x = sqrt|K| tau, whose rounding the difference magnifies by 1/x;
    and gamma^2 - 1, where the oracle rounds gamma^2 and a contracted
    multiply-add does not: 2^-53 / beta^2 of gamma beta_z and of the drift's
    phase tau / (beta Scxl)."""
    n, tau = 5003, 0.0125
    cfg = ions(n)
    want, ref = cfg["pts"].copy(), np.array(cfg["refptcl"])
    orc.physconst(cfg["freq"])
    orc.lib().orc_transfmapK(tau, strength, orc.dp(ref), orc.dp(want), n, cfg["charge"] / cfg["mass"])
    with impz.Bunch(cfg["pts"], cfg["current"], cfg["mass"], cfg["charge"], cfg["freq"],
                    cfg["refptcl"], cfg["grid"], form=form, species=True) as b:
        b.map_half(impz.elem(1, 0.1, 4, 1, [strength, -1.0, 1.0]), 0.0, 0.0, tau, 1, 0)
        got = b.download()
    got = got[np.argsort(got[:, 8])]
    tol = 1e-13
    if strength:
        tol += 4 * 2.0 ** -53 / (np.sqrt(abs(strength)) * tau)
    beta2 = 1.0 - 1.0 / cfg["refptcl"][5] ** 2
    cancel = 2.0 ** -53 / beta2
    for c in range(6):
        bound = (tol + cancel) * np.sqrt(np.mean(want[:, c] ** 2))
        if c == 4:
            bound += cancel * tau / (np.sqrt(beta2) * beams.scxl(cfg["freq"]))
        assert np.max(np.abs(got[:, c] - want[:, c])) <= bound, c


@pytest.mark.parametrize("form,cols,tol", [(impz.FORM_FP64, RMS_COLS, 1e-8),
                                           (impz.FORM_FP32CONV, FP32_COLS, 1e-5)])
def test_run_through_kmap_quadrupoles_of_two_charge_states(form, cols, tol):
    cfg = ions(20_011)
    quad = lambda k: impz.elem(1, 0.1, 4, 1, [k, -1.0, 1.0])  # noqa: E731
    drift = impz.elem(0, 0.1, 4, 1, [1.0])
    with bunch(cfg, form, species=True) as b:
        compare(b, [drift, quad(8.0), drift, quad(-8.0), quad(0.0)], cfg, cols=cols, tol=tol)


def test_group_of_different_passes_equals_solo_in_the_fp32_form():
    cfgs = [config(1000 + 777 * k) for k in range(3)]
    lats = [ORDERS["light"][:5], ORDERS["maps"][:5], ORDERS["full"][:5]]
    solo = []
    for cfg, lat in zip(cfgs, lats):
        with bunch(cfg, impz.FORM_FP32CONV) as b:
            solo.append(b.run(lat)[0])
    group = [bunch(cfg, impz.FORM_FP32CONV) for cfg in cfgs]
    for (recs, _), want in zip(impz.run_batch(group, lats), solo):
        scale = np.max(np.abs(want[:, :44]), axis=0) + 1e-300
        assert np.max(np.abs(recs[:, :44] - want[:, :44]) / scale) <= 1e-9
    for b in group:
        b.close()


def test_group_of_different_passes_equals_solo():
    cfgs = [config(1000 + 777 * k) for k in range(3)]
    for lats in ([ORDERS["light"][:5], ORDERS["maps"][:5]],
                 [ORDERS["light"][:5], ORDERS["maps"][:5], ORDERS["full"][:5]]):
        solo = []
        for cfg, lat in zip(cfgs, lats):
            with bunch(cfg) as b:
                solo.append(b.run(lat)[0])
        group = [bunch(cfg) for cfg in cfgs[:len(lats)]]
        for (recs, _), want in zip(impz.run_batch(group, lats), solo):
            scale = np.max(np.abs(want[:, :44]), axis=0) + 1e-300
            assert np.max(np.abs(recs[:, :44] - want[:, :44]) / scale) <= 1e-10
        for b in group:
            b.close()


@pytest.mark.parametrize("nz", [4, 32, 512])
@pytest.mark.parametrize("n", [65, 20_011])
def test_wake_over_few_and_many_planes(nz, n):
    """A warp meets up to 32 planes at once (the first pass over particles in
    upload order) or a single one (after the sort, few planes)."""
    pts, ref = beams.gaussian_bunch(n, seed=beams.SEED0 + 96, mass=beams.ELECTRON_MASS_EV,
                                    charge=-1.0, ekin=98.169272e6, current=1.3, freq=1.3e9,
                                    sig_x=0.5e-3, sig_y=0.5e-3, sig_xp=0.05e-3, sig_yp=0.05e-3,
                                    sig_phase_deg=1.0, sig_e=50e3)
    cfg = dict(pts=pts, refptcl=ref, current=1.3, mass=beams.ELECTRON_MASS_EV, charge=-1.0,
               freq=1.3e9, grid=(8, 8, nz))
    wake = (synthetic_table(), 1.0, True)
    with bunch(cfg) as b:
        b.wake(*wake)
        compare(b, [impz.elem(0, 0.5, 3, 1, [1.0]), impz.elem(1, 0.1, 2, 1, [10.0, 0.0, 1.0])], cfg,
                wake)
