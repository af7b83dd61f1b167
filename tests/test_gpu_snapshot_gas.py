"""Every byte of a snapshot is the solver's own: the float pairs of S_g + S0
hold zeros at gas voxels, whatever the device memory held before, and two
snapshots of one solve are equal."""
import struct
import tempfile

import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu

N, GAS = 12, 3


def _create(prec, gas):
    c = synth.small_case(N, 6, 100, n_steps=1)
    c.iter_max = 5
    nl_path = c.write(tempfile.mkdtemp(prefix="snapgas_"))
    nl = capi.read_namelist(nl_path)
    nl.N_phases = 2
    nl.Type_phases[:] = (0, 1)
    slip = capi.read_slip(nl_path.rsplit("/", 1)[0] + "/mat.sx")
    mesh = c.mesh
    phase = np.where(mesh.grain == GAS, 2, 1).astype(np.int32) if gas else mesh.phase
    return capi.Rve.create(nl, slip, mesh.euler_deg, mesh.grain, phase, prec), phase


def _state(r):
    """The state: after the 64-byte header, the descriptor, the namelist, two
    ints a voxel and the increment's record (its length and rows); before the
    macro state and the log rows of the increment in progress."""
    blob = r.snapshot()
    desc, macro, nl_size, incr = struct.unpack_from("<IIII", blob, 12)
    at = 64 + desc + nl_size + 8 * N ** 3 + incr
    at += 8 + 8 * struct.unpack_from("<q", blob, at)[0]
    return blob[at:len(blob) - 12 * 8 * 5 - macro]


@pytest.mark.parametrize("prec", [capi.PREC_MIXED_IR, capi.PREC_MIXED_NR32])
def test_gas_voxels_hold_zeros_in_a_snapshot(prec, voce_lib):
    states, kept = [], []
    for _ in range(3):
        # the memory of an RVE without gas comes back to the next one: its
        # neighbours stay, so that the allocator keeps the blocks they share
        kept.append(_create(prec, False)[0])
        r, _ = _create(prec, False)
        kept.append(_create(prec, False)[0])
        r.run(1)
        r.close()
        r, phase = _create(prec, True)
        r.run(1)
        states.append(_state(r))
        r.close()
    for r in kept:
        r.close()
    assert states[0] == states[1] == states[2]
    # 214 doubles and the phase id a voxel, then the float columns: (15 S0),
    # 24 1/CRSS, 15 S_g + S0, and the low parts of the last two
    nv = N ** 3
    first = nv * (214 * 8 + 4 + (60 if prec == capi.PREC_MIXED_NR32 else 0) + 96)
    cols = [np.frombuffer(states[0], np.float32, 15 * nv, first + k * 4 * 39 * nv).reshape(15, nv) for k in (0, 1)]
    for c in cols:
        assert np.all(c[:, phase == 2] == 0.0)
    assert np.all(cols[0][0, phase == 1] != 0.0)
