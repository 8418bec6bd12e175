"""The x-first A-product (x, then y, then z with the spectral product): every compiled length of
each axis, at its largest lattice and below it, full boxes and boxes with holes, in both
precisions against the oracle on the same grid.  Tolerances are those of the other product
tests: 1e-12 relative in FP64 (rounding of two FFTs), 1e-5 for the FP32 convolution.

The boxes pair a long axis with short ones, so each length is met in the x kernels and in the
y kernels, in the fused plane kernel and (planes that no block holds, axis lengths below 32) in
the separate y and z kernels."""
import numpy as np
import pytest

import oracle as O
import tdda
from conftest import rel
from tdda import lattice

XY = {12: (6,), 14: (7,), 15: (8,), 18: (9,), 20: (10,), 21: (11,), 24: (12,), 25: (13,), 32: (14, 16), 40: (18, 20),
      48: (22, 24), 56: (25, 28), 64: (29, 32), 80: (33, 40), 96: (41, 48), 112: (49, 56), 128: (57, 64),
      160: (66, 80), 192: (81, 96), 224: (97, 112), 256: (113, 128)}
Z = {12: (6,), 14: (7,), 15: (8,), 20: (9, 10), 21: (11,), 24: (12,), 25: (13,), 32: (14, 16), 40: (17, 20),
     48: (21, 24), 56: (25, 28), 64: (29, 32)}


def _boxes():
    """(box, grid): each x / y length as x beside a short y, and as y beside a short x, over the z lengths in turn."""
    zs = [(m, n) for m, ns in Z.items() for n in ns]
    short = [(12, 6), (14, 7), (15, 8), (20, 10), (32, 15)]
    out, k = [], 0
    for m, ns in XY.items():
        for n in ns:
            sm, sn = short[k % len(short)]
            zm, zn = zs[k % len(zs)]
            zm2, zn2 = zs[(5 * k + 3) % len(zs)]
            out.append(((n, sn, zn), (m, sm, zm)))
            out.append(((sn, n, zn2), (sm, m, zm2)))
            k += 1
    # planes too large for one block beside a long x axis, and the largest that fit
    out += [((33, 113, 32), (80, 256, 64)), ((40, 90, 31), (80, 192, 64)), ((30, 81, 21), (64, 192, 48)),
            ((29, 66, 25), (64, 160, 56)), ((16, 128, 16), (32, 256, 32))]
    return out


def test_boxes_reach_every_length():
    """The grids the boxes below name are the ones a core chooses."""
    boxes = _boxes()
    for (nx, ny, nz), grid in boxes:
        assert (lattice.fft_length(nx, False), lattice.fft_length(ny, False), lattice.fft_length(nz, True)) == grid
    assert {g[0] for _, g in boxes} >= set(XY) and {g[1] for _, g in boxes} >= set(XY)
    assert {g[2] for _, g in boxes} == set(Z)


@pytest.mark.gpu
@pytest.mark.parametrize("k", range(len(_boxes())))
def test_product_matches_the_oracle(k):
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    box, grid = _boxes()[k]
    rng = np.random.Generator(np.random.PCG64(1000 + k))
    R = lattice.bulk(*box)
    if k % 2:  # holes, dipoles in another order than the cells
        r = R.reshape(-1, 3)
        r = r[rng.random(len(r)) < 0.7]
        R = np.ascontiguousarray(r[rng.permutation(len(r))].ravel())
    mat = np.array([1.0, 4.0 + 0.1j])
    core = tdda.AProductCore(*box, R, 9.0, 530.0, mat)
    assert tuple(core.grid) == grid
    oc = O.OracleCore(*box, R, 9.0, 530.0, mat, grid=core.grid, pruned=True)
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    y = oc.Aproduct(b)
    assert rel(core.Aproduct(b), y) <= 1e-12
    y32 = core.Aproduct(b, precision=tdda.FP32_REFINE)
    assert rel(y32, y) <= 1e-5
    # the z-y-x passes on the same core (the spectrum's layout is the x-first product's)
    core.set_xpass(1)
    assert rel(core.Aproduct(b, precision=tdda.FP32_REFINE), y) <= 1e-5
    core.close()


@pytest.mark.gpu
def test_gather_tile_changes_no_result():
    """8 or 16 lines per block of the FP32 gather: the same products and refined solves, bit for bit."""
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    rng = np.random.Generator(np.random.PCG64(7))
    box = (33, 41, 9)
    R = lattice.bulk(*box)
    c = tdda.AProductCore(*box, R, 10.0, 560.0, np.array([1.0, 4.0 + 0.1j]))
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    m = tdda.DDAModel(c, (0.0, 0.0, 1.0), 1.0, (1.0, 0.0, 0.0), np.repeat(rng.random(R.size // 3), 3))
    out = []
    for tile in (0, 8, 16):
        c.set_xpass(0, tile)
        m.InitializeP()
        info = m.solve_mixed(10000, 1e-5)
        out.append((c.Aproduct(b, precision=tdda.FP32_REFINE), m.get_P(), info["inner_iterations"]))
    for y, P, it in out[1:]:
        assert np.array_equal(y, out[0][0]) and np.array_equal(P, out[0][1]) and it == out[0][2]
    m.close()
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [tdda.FP64, tdda.FP32_REFINE])
@pytest.mark.parametrize("how", ["aligned", "unaligned", "in place", "overlapping"])
def test_product_on_device_vectors_equals_the_one_on_host_vectors(how, precision):
    """Device vectors are read and written by the kernels themselves; an address that is not a
    multiple of 16 goes through the staging vectors.  Same values bit for bit, also where the
    result overwrites the operand (wholly, or one entry further on)."""
    torch = pytest.importorskip("torch")
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    box = (21, 17, 11)
    R = lattice.bulk(*box)
    c = tdda.AProductCore(*box, R, 10.0, 560.0, np.array([1.0, 4.0 + 0.1j]))
    rng = np.random.Generator(np.random.PCG64(17))
    b = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    want = c.Aproduct(b, precision=precision)
    n = 2 * R.size
    buf = torch.zeros(2 * n + 16, dtype=torch.float64, device="cuda")
    at = {"aligned": (0, n + 2), "unaligned": (1, n + 3), "in place": (0, 0), "overlapping": (0, 2)}[how]
    buf[at[0]:at[0] + n] = torch.from_numpy(b.view(np.float64))
    torch.cuda.synchronize()
    c.Aproduct_device(buf.data_ptr() + 8 * at[0], buf.data_ptr() + 8 * at[1], precision)
    got = buf[at[1]:at[1] + n].cpu().numpy().view(np.complex128)
    assert np.array_equal(got, want)
    c.close()
