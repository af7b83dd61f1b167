"""The finalisers at the end of an increment (kb_finalize): every RVE of a
batch with more members than the launch has blocks ends its last increment
with its whole macro state written.

The end of the last increment clears the RVE's active flag in the block's
shared copy of the macro state.  A thread that tested that copy after the
clearing would leave its share of the state unwritten (words of the averages,
counters and flags that follow the increment), so the state behind the last
increment is compared word by word: identical RVEs must hold identical ones,
and the one an RVE run by itself holds."""
import struct

import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu


def _macro(blob, iter_max):
    """The macro state of a snapshot: before the log rows of the increment in
    progress (12 doubles a row), which end it."""
    size, = struct.unpack_from("<I", blob, 16)
    at = len(blob) - 12 * 8 * iter_max - size
    return blob[at:at + size]


@pytest.mark.parametrize("prec", [capi.PREC_FP64, capi.PREC_MIXED_NR32])
def test_every_member_of_a_large_batch_ends_with_its_whole_macro_state(prec, voce_lib):
    mesh = synth.voronoi_mesh_box((4, 4, 4), 3, 95)
    nl, slip = capi.VoceNamelist(), capi.VoceSlip()
    m, load = synth.CU_LIKE, synth.tension_z()
    nl.CellDim[:] = mesh.dims
    nl.N_phases = 1
    nl.TimeStep, nl.N_steps, nl.IterMax, nl.Err = 0.2, 10, 3, 1e-5
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

    def create():
        return capi.Rve.create(nl, slip, mesh.euler_deg, mesh.grain, mesh.phase, prec)

    count, incs = 620, 3       # 152 x 4 blocks take the members in two turns
    with create() as r:
        r.run(incs)
        want = [r.increment(k) for k in range(incs)]
    rves = [create() for _ in range(count)]
    with capi.Batch(prec) as b:
        for r in rves:
            b.add(r, incs)
        assert b.run() == 0
        for r in rves:
            b.remove(r)
    states = set()
    for r in rves:
        assert r.increments_done == incs
        assert [r.increment(k) for k in range(incs)] == want
        states.add(_macro(r.snapshot(), nl.IterMax))
        r.close()
    assert len(states) == 1
    # its 119 leading words are averages, norms and sums
    macro = np.frombuffer(states.pop()[:8 * 119], dtype=np.float64)
    assert np.all(np.isfinite(macro))
