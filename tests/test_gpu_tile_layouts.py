"""FFT tiles that fit the passes' line buffers but not the larger layouts of
the register FFT (a long x edge over a short y edge, whose y tile is past the
two padded stream buffers, and forced tiles of the x and z passes): such an
RVE is created, and runs as with small tiles, bit for bit."""
import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _create(dims, prec, seed, mixed_load=True):
    mesh = synth.voronoi_mesh_box(dims, 9, seed)
    nl, slip = capi.VoceNamelist(), capi.VoceSlip()
    m = synth.CU_LIKE
    load = synth.tension_z() if mixed_load else \
        synth.random_traceless_load(np.random.Generator(np.random.PCG64(seed)))
    nl.CellDim[:] = mesh.dims
    nl.N_phases = 1
    nl.TimeStep, nl.N_steps, nl.IterMax, nl.Err = 0.2, 10, 6, 1e-5
    nl.Update_Flag = nl.Hard_Flag = 1
    nl.VelGrad_BC_Flag[:], nl.VelGrad_BC[:] = load.velgrad_flag, load.velgrad
    nl.Stress_BC_Flag[:], nl.Stress_BC[:] = load.stress_flag, load.stress
    nl.ElastConst_PhaseI[:] = (168400.0, 121400.0, 75400.0, 0.35)
    for k in ("self", "coplane", "cross", "glissile", "hirth", "lomer"):
        getattr(nl, k)[0] = 1.0
    slip.nsys, slip.nrs, slip.gamd0 = 12, 20.0, m.gamd0
    slip.tau0f, slip.tau0b, slip.tau1, slip.thet0, slip.thet1 = m.tau0f, m.tau0b, m.tau1, m.thet0, m.thet1
    for k, (n, b) in enumerate(synth.FCC_111_110):
        slip.bn[k][:], slip.bb[k][:] = n, b
    # the single-precision forms' timed schedules change the rounding: their
    # defaults, with the fixed-budget tiles; the FP64 form with the timed tiles
    lib = capi.load()
    lib.voce_set_autotune(int(prec == capi.PREC_FP64))
    try:
        return capi.Rve.create(nl, slip, mesh.euler_deg, mesh.grain, mesh.phase, prec)
    finally:
        lib.voce_set_autotune(1)


def _solve(r):
    r.run(2)
    return [r.increment(k) for k in range(2)], r.field("sig"), r.field("disgrad")


@pytest.mark.parametrize("dims,prec,yxt", [
    ((256, 24, 4), capi.PREC_FP64, 256),       # register FFT along y, 237568 B for the stream
    ((384, 16, 2), capi.PREC_FP64, 384),
    ((324, 18, 2), capi.PREC_FP64, 324),       # a factor 3 along y
    ((216, 32, 2), capi.PREC_FP64, 216),       # only when asked for
    ((864, 12, 2), capi.PREC_MIXED, 864),
    ((512, 24, 2), capi.PREC_MIXED_IR, 512),
])
def test_long_x_edges_over_short_y_edges(dims, prec, yxt, voce_lib):
    with _create(dims, prec, 96) as r:
        want = _solve(r)
        assert np.all(np.isfinite(want[1]))
    with _create(dims, prec, 96) as r:
        t = r.tiles()
        for ty in (yxt, 1):                    # past the stream's size, and a small one
            t[1] = ty
            r.set_tiles(t)
            assert r.tiles()[1] == ty
            with capi.Rve.restore(r.snapshot()) as q:
                got = _solve(q)
            assert got[0] == want[0]
            assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2]), ty


@pytest.mark.parametrize("dims,prec,tiles", [
    # z forward, y, x/Green, z inverse tiles, each past the register FFT's own layout
    ((64, 36, 64), capi.PREC_FP64, [36, 2, 18, 36]),
    ((144, 24, 144), capi.PREC_FP64, [8, 2, 8, 12]),      # 12 x 12
    ((8, 96, 32), capi.PREC_MIXED, [96, 2, 8, 48]),
    ((8, 72, 32), capi.PREC_MIXED_NR32, [72, 2, 8, 72]),
    ((36, 64, 8), capi.PREC_MIXED, [8, 2, 64, 8]),        # 6 x 6
])
@pytest.mark.parametrize("mixed_load", [False, True])     # with and without a mean correction of the gradient
def test_tiles_beyond_the_register_layout(dims, prec, tiles, mixed_load, voce_lib):
    with _create(dims, prec, 97, mixed_load) as r:
        assert all(r.fft_split(a) > 0 for a in range(3))
        t = r.tiles()
        got = []
        for use in (tiles, [1, 1, 1, 1]):
            r.set_tiles(use + t[4:])
            with capi.Rve.restore(r.snapshot()) as q:
                assert q.tiles() == use + t[4:]
                got.append(_solve(q))
    assert got[0][0] == got[1][0]
    assert np.all(np.isfinite(got[0][1]))
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])
