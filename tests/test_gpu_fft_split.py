"""Which transform an axis runs: the register FFT that stands in for the
default Stockham order (FP64 axes, and the lengths with 9 in every form), and
that order itself when the caller asks for it.  Both are a DFT: they agree to
rounding, 4 log2(L) ulp, and differ in their last bits."""
import math
import tempfile

import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _case(dims, seed):
    c = synth.Case("split", synth.voronoi_mesh_box(dims, 10, seed), synth.CU_LIKE, synth.tension_z(), 0.2, 1)
    return c.write(tempfile.mkdtemp(prefix="split_"))


@pytest.mark.parametrize("fp64,L", [(True, 24), (True, 64), (True, 144), (False, 18), (False, 108)])
def test_the_default_order_can_be_probed(fp64, L, voce_lib):
    rng = np.random.Generator(np.random.PCG64(L))
    x = (rng.standard_normal((9, L)) + 1j * rng.standard_normal((9, L))).astype(np.complex64)
    eps = 2.0 ** -53 if fp64 else 2.0 ** -24
    for sign in (-1, 1):
        a, b = (capi.diag_fft(x, sign, k, fp64) for k in (0, -1))
        assert not np.array_equal(a, b)
        scale = math.sqrt(np.mean(np.abs(a) ** 2))
        assert math.sqrt(np.mean(np.abs(a - b) ** 2)) <= 4 * math.log2(L) * eps * scale
    with pytest.raises(capi.VoceError):
        capi.diag_fft(x[:, :16], -1, -1, False)     # 16 in single precision: a candidate of its own


@pytest.mark.parametrize("prec,dims,splits", [
    (capi.PREC_FP64, (24, 32, 48), [4, 4, 6]),
    (capi.PREC_MIXED, (18, 12, 36), [6, 4, 6]),
])
def test_a_set_default_schedule_runs_its_stages(prec, dims, splits, voce_lib):
    nl = _case(dims, 101)
    lib = capi.load()
    lib.voce_set_autotune(0)
    try:
        r, q = (capi.Rve.from_files(nl, prec) for _ in range(2))
    finally:
        lib.voce_set_autotune(1)
    radices = [r.fft_schedule(a) for a in range(3)]
    assert [r.fft_split(a) for a in range(3)] == splits
    for a in range(3):
        q.set_fft_schedule(a, 0)
    assert [q.fft_split(a) for a in range(3)] == [0, 0, 0]
    assert [q.fft_schedule(a) for a in range(3)] == radices
    blob = q.snapshot()
    r.run(1)
    q.run(1)
    sig = [x.field("sig") for x in (r, q)]
    assert r.increment(0)["iters"] == q.increment(0)["iters"]
    assert not np.array_equal(*sig)
    tol = 1e-12 if prec == capi.PREC_FP64 else 1e-5
    assert np.abs(sig[0] - sig[1]).max() <= tol * np.abs(sig[0]).max()
    # a snapshot keeps the choice, and a tile change leaves it
    with capi.Rve.restore(blob) as p:
        assert [p.fft_split(a) for a in range(3)] == [0, 0, 0]
        p.set_tiles([1, 1, 1, 1, 1, 1])
        p.run(1)
        assert np.array_equal(p.field("sig"), sig[1])
    r.close()
    q.close()
