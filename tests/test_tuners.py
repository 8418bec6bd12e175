"""What the tuners leave on a core: they choose among products that a core may run, so the product
after a call is one of those they timed and never a form that they did not compare."""
import numpy as np
import pytest

import tdda
from tdda import lattice

MAT = np.array([1.0, 4.0 + 0.1j])


@pytest.mark.gpu
@pytest.mark.parametrize("box", [(6, 20, 10), (7, 10, 6), (9, 16, 12), (13, 13, 13), (97, 12, 9), (112, 40, 20), (128, 20, 10)])
def test_x_lengths_of_one_form_keep_their_product(box):
    """FFT x lengths without a register form of the x pass (12 to 25, 224, 256) have one candidate:
    the tuner, and either form set by hand, leave the x-first product, bit by bit."""
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    R = lattice.bulk(*box)
    c = tdda.AProductCore(*box, R, 9.0, 530.0, MAT)
    rng = np.random.Generator(np.random.PCG64(sum(box)))
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    names, y = c.pass_names(tdda.FP32_REFINE), c.Aproduct(b, precision=tdda.FP32_REFINE)
    assert names[0] == "k_xfwd"
    t = c.autotune(nrhs=1, reps=2)
    assert len(t["candidates"]) == 1
    for form in (None, 0, 1):
        if form is not None:
            c.set_xpass(form)
        assert c.pass_names(tdda.FP32_REFINE) == names
        assert np.array_equal(c.Aproduct(b, precision=tdda.FP32_REFINE), y)
    c.close()
