"""The Green spectrum from the octant of offsets and the directly summed products, by the product it gives against direct summation
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


# both sides of the direct product's limit, blocks of one and two dipoles, warps without a neighbour
BOXES += [(1, 1, 2), (3, 1, 1), (8, 8, 8), (19, 3, 9), (5, 13, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("direct", ["1", "0"])  # products of up to 512 dipoles summed directly, or by transforms
@pytest.mark.parametrize("fill", [1.0, 0.6])
@pytest.mark.parametrize("box", BOXES)
def test_product_equals_direct_summation(box, fill, direct, monkeypatch):
    monkeypatch.setenv("TDDA_DIRECT", direct)
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


@pytest.mark.gpu
@pytest.mark.parametrize("method,periodic", [("FCD", None), ("LDR", (3, 2, 180.0, 200.0))])
def test_direct_product_of_other_tensors(method, periodic, monkeypatch):
    """The directly summed product of the FCD and the periodic tensor against the transforms'."""
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    rng = np.random.Generator(np.random.PCG64(8))
    R = np.array([(x, y, z) for x in range(6) for y in range(7) for z in range(5)], np.int32)
    R = np.ascontiguousarray(R[np.sort(rng.permutation(len(R))[:150])].ravel())
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    y = []
    for direct in ("1", "0"):
        monkeypatch.setenv("TDDA_DIRECT", direct)
        core = tdda.AProductCore(6, 7, 5, R, 9.0, 540.0, np.array([1.0, 4.0 + 0.1j]), 1.0, method=method,
                                 periodic=periodic)
        y.append(core.Aproduct(b))
        core.close()
    assert rel(y[0], y[1]) <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 5, -7])
def test_direct_product_of_overlapping_device_vectors(shift):
    """Input and output in one device buffer, the same or shifted by entries: the result of separate ones."""
    torch = pytest.importorskip("torch")
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    rng = np.random.Generator(np.random.PCG64(9))
    R = np.array([(x, y, z) for x in range(8) for y in range(8) for z in range(8)], np.int32).ravel()
    core = tdda.AProductCore(8, 8, 8, R, 9.0, 540.0, np.array([1.0, 4.0 + 0.1j]), 1.0)
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    want = core.Aproduct(b)
    buf = torch.zeros(R.size + 16, dtype=torch.complex128, device="cuda")
    i, o = 8, 8 + shift
    for _ in range(5):
        buf[i:i + R.size] = torch.from_numpy(b).cuda()
        torch.cuda.synchronize()
        st = tdda.load().tdda_aproduct(core.h, tdda.FP64, buf[i:].data_ptr(), buf[o:].data_ptr(), tdda.MEM_DEVICE)
        assert st == tdda.OK
        assert np.array_equal(buf[o:o + R.size].cpu().numpy(), want)
    core.close()
