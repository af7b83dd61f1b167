"""Shared memory of the FFT passes over all edges and tiles (host arithmetic,
no GPU): a tile that fits its phase, by two line buffers of a block, is
accepted, and what the plan then asks for fits in a block as well."""
import pytest

from voce_gb300 import capi

BLOCK = 227 * 1024
EDGES = sorted(e for a in range(11) for b in range(7) if 2 <= (e := 2 ** a * 3 ** b) <= 1024)
CPLX = {capi.PREC_FP64: 16, capi.PREC_MIXED: 8}


def _divisors(n):
    return [k for k in range(1, n + 1) if n % k == 0]


def _two_line_buffers(length, lines, cplx):
    return 2 * length * (lines | 1) * cplx


@pytest.mark.parametrize("prec", sorted(CPLX))
def test_default_tiles_fit_on_every_grid(prec, voce_lib):
    for nx in EDGES:
        for ny in EDGES:
            for nz in (2, 12, 64, 144, 1024):
                assert max(capi.fft_smem((nx, ny, nz), prec)) <= BLOCK, (nx, ny, nz)


@pytest.mark.parametrize("prec", sorted(CPLX))
def test_every_y_tile_that_fits_two_line_buffers_runs(prec, voce_lib):
    tried = 0
    for nx in EDGES:
        for ny in EDGES:
            for t in _divisors(nx):
                if _two_line_buffers(ny, t, CPLX[prec]) > BLOCK:
                    with pytest.raises(capi.VoceError):
                        capi.fft_smem((nx, ny, 2), prec, [1, t, 1, 1, 1, 1])
                    break
                assert max(capi.fft_smem((nx, ny, 2), prec, [1, t, 1, 1, 1, 1])) <= BLOCK, (nx, ny, t)
                tried += 1
    assert tried > 5000


def test_tiles_are_checked_as_set_tiles_does(voce_lib):
    for bad in ([3, 1, 1, 1, 1, 1], [1, 0, 1, 1, 1, 1], [1, 1, 1, 1, 1, 5]):
        with pytest.raises(capi.VoceError):
            capi.fft_smem((8, 8, 8), capi.PREC_FP64, bad)
    with pytest.raises(capi.VoceError):
        capi.fft_smem((8, 8, 7))
