"""Shared-memory layout of the z transforms' tile copies (host arithmetic of the
library, no GPU): a TMA copy's destination must lie on 128 bytes, or the copy
faults."""
import ctypes as C

import pytest

from afid_b200 import _lib


def smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def shape(nym, nzm, fy=0, fz=0):
    t = _lib.TileShape()
    _lib.check(_lib.lib().afid_fft_tile_shape(nym, nzm, fy, fz, C.byref(t)))
    return t


@pytest.mark.parametrize("nym", [2, 4, 6, 8, 10, 14, 64, 1024])
def test_z_tile_copies_are_aligned(nym):
    for nzm in range(2, 3073):
        if not smooth(nzm):
            continue
        for fz in (0, 1, 2, 4, 8, 16, 32, 64):
            try:
                t = shape(nym, nzm, 0, fz)
            except _lib.AfidError as e:
                assert fz and e.code == -1
                continue
            line = 16 * t.z_lines            # bytes of one kz row of the tile
            assert t.z_slot * 16 % 128 == 0 and t.z_slot >= t.z_lines * nzm
            assert 1 <= t.z_rows <= min(nzm, 256)
            whole = nzm // t.z_rows          # tile copies, each on 128 bytes
            assert all(c * t.z_rows * line % 128 == 0 for c in range(whole))
            assert whole + nzm % t.z_rows <= 48   # the rest as one copy a row
            assert (2 * t.z_slot + nzm) * 16 + 1024 <= 200 * 1024


def test_tile_shape_tells_the_kernels_apart():
    for n, tile in ((384, 0), (1024, 0), (960, 0), (972, 1), (1000, 1), (98, 1), (1152, 1), (14, 1)):
        t = shape(n, n)
        assert (t.y_tile, t.z_tile) == (tile, tile), n
    assert (shape(384, 972).y_tile, shape(384, 972).z_tile) == (0, 1)
    for bad in ((10, 11), (9, 8), (22, 8), (10, 4096)):
        with pytest.raises(_lib.AfidError):
            shape(*bad)
    with pytest.raises(_lib.AfidError):
        shape(10, 972, 0, 3)
