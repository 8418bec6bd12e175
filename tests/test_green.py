"""The Green spectrum from the octant of offsets, by the product it gives against direct summation
of the tensor: axes of one cell, odd and even FFT lengths, lengths with and without compiled axis
kernels (the two layouts of the folded spectrum), a partly filled box.  Tolerance: 1e-12 of the
largest entry, that of the other FP64 products (rounding of two FFTs)."""
import math

import numpy as np
import pytest

import oracle as O
import tdda
from conftest import rel

BOXES = [(3, 2, 1), (1, 1, 33), (1, 25, 1), (130, 2, 2), (2, 150, 1), (8, 13, 7), (12, 3, 70), (11, 5, 13), (17, 6, 11)]


@pytest.mark.gpu
@pytest.mark.parametrize("fill", [1.0, 0.6])
@pytest.mark.parametrize("box", BOXES)
def test_product_equals_direct_summation(box, fill):
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    rng = np.random.Generator(np.random.PCG64(sum(box)))
    R = np.array([(x, y, z) for x in range(box[0]) for y in range(box[1]) for z in range(box[2])], np.int32)
    if fill < 1.0:
        R = R[np.sort(rng.permutation(len(R))[:max(2, int(fill * len(R)))])]
    R = np.ascontiguousarray(R.ravel())
    lam, d = 540.0, 9.0
    core = tdda.AProductCore(*box, R, d, lam, np.array([1.0, 4.0 + 0.1j]), 1.0)
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    assert rel(core.Aproduct(b), O.aproduct_direct(R, d, 2 * math.pi / lam, b)) <= 1e-12
    core.close()
