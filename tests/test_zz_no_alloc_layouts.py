"""The allocation-free product where the x-first product's work grid (3 Mx My Nz entries) exceeds the
static array and the z-first one (3 Nx My Mz) does not: the FP64 z-y-x passes on a spectrum laid out
for the x-first product.  Against direct summation, and bit by bit the same again after a grid that
takes the x-first product.  Tolerance: 1e-12 as for the other FP64 products."""
import math

import numpy as np
import pytest

import oracle as O
import tdda
from conftest import rel

pytestmark = pytest.mark.gpu
LIMIT = 4 << 20  # entries of the static array


def _core(box, n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    cells = np.unique(np.concatenate([[0, box[0] * box[1] * box[2] - 1], rng.integers(0, box[0] * box[1] * box[2], n)]))
    R = np.stack([cells // (box[1] * box[2]), cells // box[2] % box[1], cells % box[2]], axis=1).astype(np.int32)
    R = np.ascontiguousarray(R[rng.permutation(len(R))].ravel())
    core = tdda.AProductCore(*box, R, 9.0, 540.0, np.array([1.0, 4.0 + 0.1j]), 1.0)
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    return core, b, O.aproduct_direct(R, 9.0, 2 * math.pi / 540.0, b)


@pytest.mark.parametrize("box", [(97, 97, 32), (97, 112, 32), (81, 113, 32), (83, 120, 31)])
def test_passes_on_the_x_first_spectrum(box):
    torch = pytest.importorskip("torch")
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    core, b, want = _core(box, 700, sum(box))
    small, bs, _ = _core((20, 20, 10), 900, 1)
    mx, my, mz = core.grid
    assert 3 * box[0] * my * mz <= LIMIT < 3 * mx * my * box[2]
    got = []
    for c, v in ((core, b), (small, bs), (core, b)):
        vd = torch.from_numpy(v).cuda()
        yd = torch.empty_like(vd)
        torch.cuda.synchronize()
        c.Aproduct_noalloc(vd.data_ptr(), yd.data_ptr())
        got.append(yd.cpu().numpy())
    assert rel(got[0], want) <= 1e-12
    assert np.array_equal(got[0], got[2])
    assert rel(core.Aproduct(b), want) <= 1e-12
    core.close()
    small.close()
