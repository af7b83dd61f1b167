"""Values that are not finite stay visible: in the device's conversions
between double and float, and through the solver in every form, where a
stress or a load that is NaN or infinite must not come out as ordinary
numbers (the reference computes in double throughout and spreads them,
evolution.c:350-394)."""
import struct
import tempfile

import numpy as np
import pytest

from voce_gb300 import capi, synth

pytestmark = pytest.mark.gpu

FORMS = [capi.PREC_FP64, capi.PREC_MIXED, capi.PREC_MIXED_NR32, capi.PREC_MIXED_IR]


def test_conversions_over_the_whole_double_range(voce_lib):
    rng = np.random.Generator(np.random.PCG64(17))
    m = 1.0 + rng.random(8)
    x = np.concatenate([np.ldexp(m, e) for e in range(-1074, 1024)] +
                       [[0.0, 5e-324, 2.0 ** -149, 2.0 ** -150, 2.0 ** -126, 2.0 ** 128, np.inf, np.nan,
                         np.nextafter(2.0 ** -126, 0.0), np.nextafter(2.0 ** 128, 0.0),
                         float(np.finfo(np.float32).max), 1.7976931348623157e308]])
    x = np.concatenate([x, -x])
    rn, back, pair, head = capi.diag_convert(x)
    with np.errstate(over="ignore"):
        f = x.astype(np.float32)
    lo, hi = 2.0 ** -126, 2.0 ** 128
    big = ~(np.abs(x) < hi)                                    # NaN, infinity, beyond the floats
    assert not np.isfinite(rn[big]).any()
    assert not np.isfinite(back[~np.isfinite(f)]).any()
    small = np.abs(x) < lo
    assert (np.abs(rn[small]) <= lo).all() and np.all(rn[x == 0.0] == 0.0)
    n = ~big & ~small
    fn = f[n].astype(np.float64)
    assert n.sum() > 2000
    assert np.array_equal(rn[n], fn)                           # (no value is a tie)
    normal = np.isfinite(f) & (np.abs(f) >= lo)
    assert np.array_equal(back[normal], f[normal].astype(np.float64))
    assert np.all(back[np.abs(f) < lo] == 0.0)
    s = ~np.isnan(x)
    assert np.array_equal(np.signbit(rn[s]), np.signbit(x[s]))
    # the float pair: the nearest float, and a remainder (at most 2^-24 of x's
    # power of two) rounded to a float's 24 bits
    p = (np.abs(x) >= 2.0 ** -74) & (np.abs(x) < np.nextafter(hi, 0.0))
    assert np.array_equal(head[p], f[p].astype(np.float64))
    assert np.all(np.abs(pair[p] - x[p]) <= 2.0 ** -49 * np.abs(x[p]))


def test_a_tie_rounds_away_from_zero(voce_lib):
    x = np.array([1.0 + 2.0 ** -24, -1.0 - 3 * 2.0 ** -24, 2.0 - 2.0 ** -24])
    rn, _, pair, head = capi.diag_convert(x)
    assert head.tolist() == rn.tolist() and pair.tolist() == x.tolist()
    assert rn.tolist() == [1.0 + 2.0 ** -23, -1.0 - 2.0 ** -22, 2.0]


def _case(seed, iter_max):
    c = synth.small_case(8, 5, seed, n_steps=1)
    c.iter_max = iter_max
    return c.write(tempfile.mkdtemp(prefix="nonfinite_"))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("prec", FORMS)
def test_one_stress_that_is_not_finite_reaches_the_whole_spectrum(prec, bad, voce_lib):
    """A snapshot with one stress component of one voxel replaced: after one
    Green iteration no voxel's displacement gradient or stress is finite, and
    the records say so."""
    nl = _case(98, 1)
    with capi.Rve.from_files(nl, prec) as r:
        blob = bytearray(r.snapshot())
    # the state follows the 64-byte header, the descriptor, the namelist and
    # two ints a voxel; the stress comes first (component-major, 512 voxels)
    desc_size, _, nl_size = struct.unpack_from("<III", blob, 12)
    at = 64 + desc_size + nl_size + 8 * 512
    struct.pack_into("<d", blob, at + 8 * (2 * 512 + 77), bad)
    with capi.Rve.restore(bytes(blob)) as r:
        r.run(1)
        assert not np.isfinite(r.field("disgrad")).all(axis=1).any()
        assert not np.isfinite(r.field("sig")).all(axis=1).any()
        rec = r.increment(0)
        assert np.isnan(rec["s_vm"])
        assert np.isnan(np.array(rec["sig_avg"])).any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("prec", FORMS)
def test_a_load_that_is_not_finite_gives_no_finite_stress(prec, bad, voce_lib):
    nl_path = _case(99, 4)
    nl = capi.read_namelist(nl_path)
    nl.VelGrad_BC[2] = bad
    slip = capi.read_slip(nl_path.rsplit("/", 1)[0] + "/mat.sx")
    mesh = synth.small_case(8, 5, 99, n_steps=1).mesh
    with capi.Rve.create(nl, slip, mesh.euler_deg, mesh.grain, mesh.phase, prec) as r:
        r.run(1)
        assert not np.isfinite(r.field("sig")).all(axis=1).any()
        assert not np.isfinite(r.increment(0)["s_vm"])
