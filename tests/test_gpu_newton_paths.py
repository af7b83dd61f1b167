"""Branches of the Newton solves that the usual inputs do not take: exponents
above 20 and resolved-shear ratios past 60 in the crystal-axes kernels (their
correction is then solved in FP64), the switches of the general kernels that
run every slip table off the {111}<110> family, and the mixed_nr32 form's
stress, orientation and CRSS.

The general path is reached as in test_gpu_fcc.py, by a relative shift of one
component of every plane normal.  Shifted by 1.5e-11, the Schmid tensors move
by as much and the strain rate by at most n = 40 times that, 6e-10: under the
1e-9 of the FP64 form."""
import numpy as np
import pytest

import golden_io as gio
from test_gpu_fcc import TOL, _namelist, _slip
from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu

PLAIN = (range(12), [(1, 1)] * 12)


def _run(prec, nl, slip, mesh, n):
    with capi.Rve.create(nl, slip, mesh.euler_deg, mesh.grain, mesh.phase, prec) as r:
        r.run(n)
        inc = [r.increment(k) for k in range(n)]
        return inc, {f: r.field(f) for f in ("sig", "edot", "gamdot", "crss", "tranmat")}


@pytest.mark.parametrize("prec", sorted(TOL))
@pytest.mark.parametrize("nrs,tau,gamd0", [
    (25.0, None, None),        # above 20: |r|^(n-1) past the float pairs' range
    (40.0, None, None),
    (1.0, 0.05, 1e-6),         # ratios of some hundreds
    (3.0, 0.2, 1e-9),
])
def test_corrections_solved_in_fp64(prec, nrs, tau, gamd0, voce_lib):
    rng = np.random.Generator(np.random.PCG64(140))
    mesh = synth.voronoi_mesh_box((8, 6, 8), 7, 141)
    nl = _namelist(mesh.dims, synth.random_traceless_load(rng), 40)
    out = []
    for shift in (0.0, 1.5e-11):
        s = _slip(*PLAIN, shift, nrs)
        if tau is not None:
            s.tau0f = s.tau0b = tau
            s.gamd0 = gamd0
        out.append(_run(prec, nl, s, mesh, 3))
    (inc, a), (inc0, b) = out
    if tau is not None:   # rate = gamd0 r^n
        assert np.abs(a["gamdot"]).max() > gamd0 * 60.0 ** nrs
    for f in a:
        assert np.all(np.isfinite(a[f]))
        assert np.abs(a[f] - b[f]).max() <= TOL[prec] * np.abs(b[f]).max(), f
    slack = 0 if prec in (capi.PREC_FP64, capi.PREC_MIXED) else 1
    assert all(abs(x["iters"] - y["iters"]) <= slack for x, y in zip(inc, inc0))


def _off_family(prec, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    mesh = synth.voronoi_mesh_box((8, 8, 8), 7, seed)
    nl = _namelist(mesh.dims, synth.random_traceless_load(rng), 60)
    return _run(prec, nl, _slip(*PLAIN, 1e-3), mesh, 3)


def test_chord_steps_off_the_family(voce_lib):
    """The switch changes the Newton counts there, and the results by no more
    than a chord step may."""
    lib = capi.load()
    lib.voce_set_newton_chord(0)
    try:
        exact = _off_family(capi.PREC_MIXED, 142)
    finally:
        lib.voce_set_newton_chord(1)
    chord = _off_family(capi.PREC_MIXED, 142)
    assert [x["nr_iters_total"] for x in chord[0]] != [x["nr_iters_total"] for x in exact[0]]
    for a, b in zip(chord[0], exact[0]):
        assert abs(a["iters"] - b["iters"]) <= 1
        assert gio.rel(a["sig_avg"], b["sig_avg"]) < 1e-7
    assert gio.rel(chord[1]["sig"], exact[1]["sig"]) < 1e-6
    assert gio.rel(chord[1]["edot"], exact[1]["edot"]) < 1e-6


def test_float_jacobian_off_the_family(voce_lib):
    """mixed_ir with and without its start against the exact-Jacobian Newton
    of the mixed form, with the general kernels."""
    lib = capi.load()
    lib.voce_set_newton_chord(0)
    try:
        exact = _off_family(capi.PREC_MIXED, 143)
    finally:
        lib.voce_set_newton_chord(1)
    runs = []
    for pred in (0, 1):
        lib.voce_set_ir_predictor(pred)
        try:
            runs.append(_off_family(capi.PREC_MIXED_IR, 143))
        finally:
            lib.voce_set_ir_predictor(1)
    assert [x["nr_iters_total"] for x in runs[0][0]] != [x["nr_iters_total"] for x in runs[1][0]]
    for inc, out in runs:
        for a, b in zip(inc, exact[0]):
            assert abs(a["iters"] - b["iters"]) <= 1
            assert gio.rel(a["sig_avg"], b["sig_avg"]) < 1e-7
        assert gio.rel(out["sig"], exact[1]["sig"]) < 1e-6
        assert gio.rel(out["edot"], exact[1]["edot"]) < 1e-5


def test_nr32_stress_orientation_and_crss(voce_lib):
    """A point taken in single precision alone is off by a few 1e-6 of the
    stress, its rate by n times that, 2e-4.  Four increments of 2e-4 strain
    then move CRSS (about 1 % an increment) by under 1e-5 and the orientation
    (rotations near 1e-3) by under 1e-6."""
    rng = np.random.Generator(np.random.PCG64(144))
    mesh = synth.voronoi_mesh_box((8, 8, 8), 7, 145)
    nl = _namelist(mesh.dims, synth.random_traceless_load(rng), 60)
    a, b = (_run(capi.PREC_MIXED_NR32, nl, _slip(*PLAIN, s), mesh, 4)[1] for s in (0.0, 4e-11))
    for f, tol in (("sig", 1e-5), ("crss", 1e-5), ("tranmat", 1e-6)):
        assert np.abs(a[f] - b[f]).max() <= tol * np.abs(b[f]).max(), f
