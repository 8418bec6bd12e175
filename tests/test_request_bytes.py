"""tdda_request_bytes by its parts, on the host: what a core allocates when it is made (its work grids
in the layout that runs, the scratch of the Green spectrum's passes, the table of direct products)."""
import numpy as np
import pytest

import tdda
from tdda import lattice

XY = {12, 14, 15, 18, 20, 21, 24, 25, 32, 40, 48, 56, 64, 80, 96, 112, 128, 160, 192, 224, 256}
Z = {12, 14, 15, 20, 21, 24, 25, 32, 40, 48, 56, 64}


@pytest.mark.parametrize("nrhs", [1, 2, 8])
@pytest.mark.parametrize("box", [(1, 1, 2), (8, 7, 5), (13, 13, 13), (97, 97, 32), (128, 128, 32), (64, 64, 4), (100, 8, 8),
                                 (20, 4, 4), (45, 33, 19), (300, 5, 70)])
def test_parts(box, nrhs):
    nx, ny, nz = box
    n = nx * ny * nz
    m = lattice.fft_length(nx, False), lattice.fft_length(ny, False), lattice.fft_length(nz, True)
    hx, hy, hz = (k // 2 + 1 for k in m)
    axes = m[0] in XY and m[1] in XY and m[2] in Z
    grid = 3 * m[1] * max(nx * m[2], m[0] * nz if axes else 0) * nrhs
    direct = n <= (512 if axes else 800) and n <= 8192
    core = (4 * n + 12 * n + 40 * 6 * hx * hy * hz + 24 * grid + 2 * 24 * 3 * n + 16 * 6 * nx * hz * (ny + hy)
            + (16 * 6 * n if direct else 0))
    model = 3 * n * (12 * 16 + 8 + 10 * 8)
    got = tdda.request_bytes(nx, ny, nz, n, nrhs)
    assert core + nrhs * model <= got <= core + nrhs * model + 2e6


@pytest.mark.parametrize("nrhs", [1, 2, 4, 8])
@pytest.mark.parametrize("box", [(8, 7, 5), (97, 97, 32), (128, 128, 32), (64, 64, 4), (100, 8, 8), (66, 81, 32), (40, 40, 12)])
def test_no_more_than_for_the_z_first_layout(box, nrhs):
    """With a full padded grid of scratch and the z-first work grid, which the estimate was made for,
    a request took this much; the x-first product's larger work grid fits in what the scratch gave
    back, so that no request of a budget that it fitted is refused."""
    nx, ny, nz = box
    n = nx * ny * nz
    m = lattice.fft_length(nx, False), lattice.fft_length(ny, False), lattice.fft_length(nz, True)
    h = np.prod([k // 2 + 1 for k in m])
    then = 4 * n + 12 * n + 40 * 6 * h + 24 * 3 * nx * m[1] * m[2] * nrhs + 48 * 3 * n + 96 * np.prod(m) + 1e6
    assert tdda.request_bytes(nx, ny, nz, n, nrhs) <= then + nrhs * 3 * n * 280
