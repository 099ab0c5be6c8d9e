"""Byte offsets of grids around 2^29 cells and faces, the largest a 32-bit byte
offset reaches: ideal-hydro runs of that size fit the device.  The offsets are
formed on the host by the kernels' own functions, nothing is allocated."""
import os

import pytest

from echo_gpu import lib as L

B = 1 << 29
GRIDS = [
    # just below, at and above the limit in cells, in x, y and eta faces, and
    # twice it
    (B - 1, 1, 1), (B, 1, 1), (B + 1, 1, 1), (2 * B, 1, 1), (1, B - 1, 1), (1, B, 1), (1, 1, B),
    (23170, 23170, 1), (23169, 23171, 1), (23171, 23171, 1), (32768, 16384, 1), (32768, 16383, 1), (3, B // 3, 1),
    (813, 813, 812), (811, 812, 813), (1024, 1024, 512), (1023, 1024, 512), (97, 97, 81),
]


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("n", GRIDS, ids=lambda n: "x".join(map(str, n)))
def test_offsets_do_not_wrap(n, exact):
    if not os.path.exists(L.library_path(exact)):
        pytest.skip("library not built")
    nx, ny, nz = n
    cells, fx = nx * ny * nz, (nx + 1) * ny * nz
    fy, fz = nx * (ny + 1) * nz, nx * ny * (nz + 1)
    off = L.unit_offsets(nx, ny, nz, exact)
    assert off[0] == off[4] == 8 * (cells - 1)
    # the faces of the directions the grid extends in
    for got, faces, m in zip(off[1:4], (fx, fy, fz), n):
        if m > 1:
            assert got == 8 * (faces - 1)
