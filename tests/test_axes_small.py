"""The boxes of test_axes.py whose plain FP64 products are summed directly, through the transforms."""
import numpy as np
import pytest

import oracle as O
import tdda
from conftest import rel
from tdda import lattice
from test_axes import _boxes


@pytest.mark.gpu
@pytest.mark.parametrize("box", sorted({b for b, _ in _boxes() if b[0] * b[1] * b[2] <= 900}))
def test_transforms_of_small_boxes(box, monkeypatch):
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    monkeypatch.setenv("TDDA_DIRECT", "0")
    R = lattice.bulk(*box)
    core = tdda.AProductCore(*box, R, 9.0, 540.0, np.array([1.0, 4.0 + 0.1j]), 1.0)
    rng = np.random.Generator(np.random.PCG64(sum(box)))
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    assert rel(core.Aproduct(b), O.aproduct_direct(R, 9.0, 2 * np.pi / 540.0, b)) <= 1e-12
    core.close()
