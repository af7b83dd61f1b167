"""Shared memory of the FFT passes over all edges and tiles (host arithmetic,
no GPU): a tile that fits its phase, by two line buffers of a block, is
accepted, and what the plan then asks for fits in a block as well."""
import pytest

from voce_gb300 import capi

BLOCK = 227 * 1024
EDGES = sorted(e for a in range(11) for b in range(7) if 2 <= (e := 2 ** a * 3 ** b) <= 1024)
# x edges whose single-precision Green pass has always run in its own layout
XG32 = (16, 24, 32, 48, 64, 96, 128, 192, 256)
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


def _staged_z(length, rows):
    """The single-precision z passes through fft_lines: bytes of the forward
    and of the inverse one (line buffers, staged runs and columns)."""
    lines, run = 8 * length * ((3 * rows) | 1), 48 * rows * length
    return lines + max(lines, run), lines + max(lines, 48 * (length // 2 + 1) * rows) + run


@pytest.mark.parametrize("prec", sorted(CPLX))
def test_every_z_and_x_tile_that_fits_the_line_buffers_is_accepted(prec, voce_lib):
    """... on the register FFT too, whose own layout is larger: the pass then
    runs on the line buffers."""
    beyond = 0
    c = CPLX[prec]
    for ny in (64, 72, 96, 144, 192, 384, 432):
        for t in _divisors(ny):
            for edge in EDGES:
                if edge % 2 == 0:
                    z = [_two_line_buffers(edge, 3 * t, c)] * 2 if c == 16 else _staged_z(edge, t)
                    for at, k, need in ((0, 0, z[0]), (3, 3, z[1])):
                        if need <= BLOCK:
                            tiles = [1] * 6
                            tiles[at] = t
                            assert capi.fft_smem((4, ny, edge), prec, tiles)[k] <= BLOCK, (ny, t, edge)
                            beyond += capi.fft_smem((4, ny, edge), prec, tiles)[k] == need
                need = _two_line_buffers(edge, 6 * t, c)
                if need <= BLOCK and not (c == 8 and edge in XG32):
                    assert capi.fft_smem((edge, ny, 4), prec, [1, 1, t, 1, 1, 1])[2] <= BLOCK, (ny, t, edge)
    assert beyond > 50


def test_the_green_tiles_of_the_single_precision_lengths_keep_their_limit(voce_lib):
    """32 points along x: 12 t (32 + 4 + 1) complex floats."""
    assert capi.fft_smem((32, 64, 4), capi.PREC_MIXED, [1, 1, 64, 1, 1, 1])[2] == 96 * 64 * 37
    with pytest.raises(capi.VoceError):
        capi.fft_smem((32, 72, 4), capi.PREC_MIXED, [1, 1, 72, 1, 1, 1])


def test_tiles_are_checked_as_set_tiles_does(voce_lib):
    for bad in ([3, 1, 1, 1, 1, 1], [1, 0, 1, 1, 1, 1], [1, 1, 1, 1, 1, 5]):
        with pytest.raises(capi.VoceError):
            capi.fft_smem((8, 8, 8), capi.PREC_FP64, bad)
    with pytest.raises(capi.VoceError):
        capi.fft_smem((8, 8, 7))
