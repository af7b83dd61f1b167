"""Every length of the register FFT, in both precisions: the line transform
against a DFT in extended precision, and the three passes of a solve against
the Stockham stages.

Bounds.  A line: 2.5 roundings a level of the transform, RMS over RMS, as the
single-precision candidates are held to (2.5 x 2^-24 = 1.5e-7, 2.5 x 2^-53 =
2.8e-16, times log2 L).  A solve: the FP64 schedules agree to 1e-12, the
single-precision ones to 1e-5."""
import math
import tempfile

import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu

LENGTHS = [8, 12, 16, 18, 24, 27, 32, 36, 48, 54, 64, 72, 81, 96, 108, 128, 144, 192, 256]


def _dft(x, sign):
    """Rows of x transformed in extended precision."""
    L = x.shape[1]
    k = (np.outer(np.arange(L), np.arange(L)) % L).astype(np.longdouble)
    a = sign * 2 * k * (4 * np.arctan(np.longdouble(1))) / L
    c, s = np.cos(a), np.sin(a)
    re, im = x.real.astype(np.longdouble), x.imag.astype(np.longdouble)
    return (re @ c - im @ s).astype(np.float64) + 1j * (re @ s + im @ c).astype(np.float64)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("L", LENGTHS)
def test_line_transform(L, fp64, voce_lib):
    n = min(7, (200 * 1024) // (32 * L) - 1)
    rng = np.random.Generator(np.random.PCG64(L))
    x = (rng.standard_normal((n, L)) + 1j * rng.standard_normal((n, L))).astype(np.complex64)
    tol = 2.5 * math.log2(L) * (2.0 ** -53 if fp64 else 2.0 ** -24)
    # -1: the stages of the default order, where the register FFT stands in for it
    for k in (0, -1) if fp64 or L not in (16, 24, 32, 48, 64, 96, 128, 192, 256) else (0,):
        for sign in (-1, 1):
            want = _dft(x, sign)
            got = capi.diag_fft(x, sign, k, fp64)
            e = math.sqrt(np.mean(np.abs(got - want) ** 2) / np.mean(np.abs(want) ** 2))
            assert e < tol, (L, k, sign, e, tol)


@pytest.mark.parametrize("prec,tol", [(capi.PREC_FP64, 1e-12), (capi.PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("dims", [(27, 54, 18), (81, 72, 36), (8, 108, 54), (144, 8, 72), (54, 27, 108), (72, 81, 8),
                                  (108, 12, 144), (12, 144, 8), (18, 36, 12)])
def test_passes_of_a_solve(dims, prec, tol, voce_lib):
    c = synth.Case("lengths", synth.voronoi_mesh_box(dims, 12, 130), synth.CU_LIKE, synth.tension_z(), 0.2, 1)
    c.iter_max = 4
    nl = c.write(tempfile.mkdtemp(prefix="lengths_"))
    lib = capi.load()
    lib.voce_set_autotune(0)
    try:
        out = []
        for stages in (False, True):
            with capi.Rve.from_files(nl, prec) as r:
                for a in range(3):
                    if stages:
                        r.set_fft_schedule(a, 0)
                    assert (r.fft_split(a) == 0) == stages
                r.run(1)
                out.append((r.field("sig"), r.field("disgrad")))
    finally:
        lib.voce_set_autotune(1)
    for a, b in zip(*out):
        assert np.all(np.isfinite(a))
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
