"""The Newton solve in crystal axes, which an RVE takes when its slip table is
the {111}<110> family in any order and with any signs, against the general
Newton with stored Schmid vectors.

The general path is reached with the same table moved off the family by a
relative 4e-11 in one component of every plane normal.  That moves the Schmid
tensors by a few 1e-11, the converged stress by as much, and the strain rate
(power n = 20) by some 20 times that: below the 1e-9 bound the FP64 form is
held to against the reference.  The forms with a single-precision spectrum are
held to what separates them from the FP64 form: mixed (FP64 Newton) ten
single-precision roundings, 1e-6; mixed_ir, whose strain rate is evaluated at
the start of its FP64 steps, the 1e-5 it keeps to an exact-Jacobian Newton;
mixed_nr32, where an increment that ends at IterMax may end on a solution in
single precision alone (a few 1e-6), n = 20 times that for the rates, 2e-4."""
import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu

TOL = {capi.PREC_FP64: 1e-9, capi.PREC_MIXED: 1e-6, capi.PREC_MIXED_IR: 1e-5, capi.PREC_MIXED_NR32: 2e-4}


def _slip(order, signs, shift=0.0, nrs=20.0, tau_back=None):
    m = synth.CU_LIKE
    s = capi.VoceSlip()
    s.nsys, s.nrs, s.gamd0 = 12, nrs, m.gamd0
    s.tau0f, s.tau0b = m.tau0f, m.tau0b if tau_back is None else tau_back
    s.tau1, s.thet0, s.thet1 = m.tau1, m.thet0, m.thet1
    for k, (o, (sn, sb)) in enumerate(zip(order, signs)):
        n, b = synth.FCC_111_110[o]
        for i in range(3):
            s.bn[k][i], s.bb[k][i] = sn * n[i], sb * b[i]
        s.bn[k][0] *= 1.0 + shift
    return s


def _namelist(dims, load, iter_max):
    nl = capi.VoceNamelist()
    nl.CellDim[:] = dims
    nl.N_phases = 2
    nl.Type_phases[:] = (0, 1)
    nl.TimeStep, nl.N_steps, nl.IterMax, nl.Err = 0.2, 10, iter_max, 1e-5
    nl.Update_Flag = nl.Hard_Flag = 1
    nl.VelGrad_BC_Flag[:], nl.VelGrad_BC[:] = load.velgrad_flag, load.velgrad
    nl.Stress_BC_Flag[:], nl.Stress_BC[:] = load.stress_flag, load.stress
    nl.ElastConst_PhaseI[:] = (168400.0, 121400.0, 75400.0, 0.35)
    for k in ("self", "coplane", "cross", "glissile", "hirth", "lomer"):
        getattr(nl, k)[0] = 1.0 + 0.1 * len(k)
    return nl


def _solve(prec, nl, slip, mesh, n):
    with capi.Rve.create(nl, slip, mesh.euler_deg, mesh.grain, mesh.phase, prec) as r:
        r.run(n)
        inc = [r.increment(k) for k in range(n)]
        out = {f: r.field(f) for f in ("sig", "edot", "gamdot", "taux", "crss", "tranmat", "svm", "evm",
                                       "rho_rss", "rho_crss", "work_p", "gammatotal")}
    return inc, out


@pytest.mark.parametrize("prec", sorted(TOL))
@pytest.mark.parametrize("dims,nrs,tau_back,shuffle", [
    ((8, 8, 8), 20.0, None, False),       # one partial work split, the exponent's product chain
    ((4, 6, 12), 7.0, 15.0, True),        # 288 voxels (a remainder), binary powering, uneven CRSS directions
    ((18, 16, 16), 20.0, 13.0, True),     # several units per block row, gas voxels
    ((2, 2, 2), 1.0, None, True),         # fewer voxels than a warp, a linear flow rule
])
def test_crystal_axes_newton_against_the_general_one(prec, dims, nrs, tau_back, shuffle, voce_lib):
    rng = np.random.Generator(np.random.PCG64(91))
    order = rng.permutation(12) if shuffle else np.arange(12)
    signs = rng.choice([-1, 1], (12, 2)) if shuffle else np.ones((12, 2), dtype=int)
    mesh = synth.voronoi_mesh_box(dims, 7, 92)
    if dims[0] == 18:
        mesh.phase[mesh.grain == 3] = 2
    nl = _namelist(dims, synth.random_traceless_load(rng), 60)
    n = 4                                  # through reorientation (2) and hardening (3)
    inc, out = _solve(prec, nl, _slip(order, signs, 0.0, nrs, tau_back), mesh, n)
    inc0, out0 = _solve(prec, nl, _slip(order, signs, 4e-11, nrs, tau_back), mesh, n)
    slack = 0 if prec in (capi.PREC_FP64, capi.PREC_MIXED) else 1
    assert all(abs(x["iters"] - y["iters"]) <= slack for x, y in zip(inc, inc0))
    for f, a in out.items():
        b = out0[f]
        assert np.all(np.isfinite(a))
        assert np.abs(a - b).max() <= TOL[prec] * max(np.abs(b).max(), 1e-300), f
    for a, b in zip(inc, inc0):
        for k in ("sig_avg", "eps_avg", "edot_avg"):
            assert np.abs(np.array(a[k]) - b[k]).max() <= TOL[prec] * np.abs(b[k]).max(), k


@pytest.mark.parametrize("prec", sorted(TOL))
def test_batch_of_both_newton_paths(prec, voce_lib):
    """A batch that mixes RVEs of the family with one off it gives each the
    bits it has alone."""
    rng = np.random.Generator(np.random.PCG64(93))
    meshes = [synth.voronoi_mesh_box(d, 5, 94 + k) for k, d in enumerate([(8, 8, 8), (6, 4, 8), (12, 8, 8)])]
    nls = [_namelist(m.dims, synth.random_traceless_load(rng), 40) for m in meshes]
    plain = [(k, np.ones(2, dtype=int)) for k in range(12)]
    slips = [_slip([p[0] for p in plain], [p[1] for p in plain], s) for s in (0.0, 1e-3, 0.0)]
    alone = [_solve(prec, nl, s, m, 2) for nl, s, m in zip(nls, slips, meshes)]
    rves = [capi.Rve.create(nl, s, m.euler_deg, m.grain, m.phase, prec)
            for nl, s, m in zip(nls, slips, meshes)]
    with capi.Batch(prec) as b:
        for r in rves:
            b.add(r, 2)
        assert b.run() == 0
        for r in rves:
            b.remove(r)
    for r, (inc, out) in zip(rves, alone):
        assert [r.increment(k) for k in range(2)] == inc
        for f in ("sig", "edot", "gamdot"):
            assert np.array_equal(r.field(f), out[f])
        r.close()
