"""The y pass streams where every RVE of a plan runs the register FFT along y,
and otherwise runs a tile at a time: an RVE alone (streamed) and in a batch
with one whose y edge has no register FFT (not streamed) gives the same bits,
for y edges with and without a factor 3."""
import tempfile

import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu

DIMS = [(8, 12, 8), (4, 18, 6), (6, 27, 4), (4, 24, 8), (4, 16, 4), (4, 81, 2), (4, 144, 2)]
UNSTREAMED = (4, 6, 8)


def _create(dims, seed, prec):
    c = synth.Case("ystream", synth.voronoi_mesh_box(dims, 5, seed), synth.CU_LIKE, synth.tension_z(), 0.2, 2)
    c.iter_max = 20
    return capi.Rve.from_files(c.write(tempfile.mkdtemp(prefix="ystream_")), prec)


@pytest.mark.parametrize("prec", [capi.PREC_FP64, capi.PREC_MIXED, capi.PREC_MIXED_IR])
def test_streamed_and_unstreamed_y_passes_agree(prec, voce_lib):
    lib = capi.load()
    lib.voce_set_autotune(0)                  # the default transforms
    try:
        alone = []
        for k, dims in enumerate(DIMS):
            with _create(dims, 110 + k, prec) as r:
                assert r.fft_split(1) > 0
                r.run(2)
                alone.append(([r.increment(i) for i in range(2)], r.field("sig"), r.field("disgrad")))
        rves = [_create(dims, 110 + k, prec) for k, dims in enumerate(DIMS)] + [_create(UNSTREAMED, 120, prec)]
    finally:
        lib.voce_set_autotune(1)
    assert rves[-1].fft_split(1) == 0
    with capi.Batch(prec) as b:
        for r in rves:
            b.add(r, 2)
        assert b.run() == 0
        for r in rves:
            b.remove(r)
    for r, (inc, sig, dg) in zip(rves, alone):
        assert [r.increment(i) for i in range(2)] == inc
        assert np.array_equal(r.field("sig"), sig) and np.array_equal(r.field("disgrad"), dg)
    for r in rves:
        r.close()
