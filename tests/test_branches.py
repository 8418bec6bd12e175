"""The FP32 steps of a batch as parallel branches of the solve's graph: each solution is, bit by
bit, the one of the right-hand side solved alone (no tolerance: the branches only divide the
batch), for one to four branches, equal and unequal shares, with the device-side loop and with
host-launched chunks."""
import numpy as np
import pytest

import tdda
from tdda import lattice

# box, right-hand sides: the number of branches their x length and count lead to on 152 SMs
CASES = [((20, 20, 10), 3, 1), ((48, 6, 6), 2, 2), ((48, 6, 6), 7, 2), ((48, 6, 6), 3, 3), ((20, 20, 10), 5, 4),
         ((20, 20, 10), 8, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("loop", ["1", "0"])
@pytest.mark.parametrize("box,n,branches", CASES)
def test_batch_equals_alone(box, n, branches, loop, monkeypatch):
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    monkeypatch.setenv("TDDA_DEVICE_LOOP", loop)
    rng = np.random.Generator(np.random.PCG64(n))
    R = lattice.bulk(*box)
    core = tdda.AProductCore(*box, R, 10.0, 520.0, np.array([1.0, 4.0 + 0.1j]), max_rhs=n)
    inc = (list(lattice.config(3).incidences) * 2)[:n]
    rho = [np.repeat(rng.random(R.size // 3), 3) for _ in range(n)]  # a density each: they stop at different steps
    ms = [tdda.DDAModel(core, i.nK, i.E0, i.nE0, d) for i, d in zip(inc, rho)]
    infos = tdda.solve_batch(ms, tdda.FP32_REFINE, 400, 1e-9)
    batch = [m.get_P() for m in ms]
    for k, m in enumerate(ms):
        m.InitializeP()
        [alone] = tdda.solve_batch([m], tdda.FP32_REFINE, 400, 1e-9)
        assert alone["inner_iterations"] == infos[k]["inner_iterations"]
        assert np.array_equal(m.get_P(), batch[k])
    for m in ms:
        m.close()
    core.close()


@pytest.mark.gpu
def test_cross_lattice_models_of_one_core_equal_alone():
    """The residuals of a cross-lattice batch run together where the cores differ and in turn where
    models share one: two models of one core beside one of another, bit by bit as alone."""
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    rng = np.random.Generator(np.random.PCG64(5))
    inc = lattice.config(3).incidences
    cores, ms = [], []
    for box, count in (((20, 20, 10), 2), ((18, 19, 9), 1)):
        R = lattice.bulk(*box)
        cores.append(tdda.AProductCore(*box, R, 10.0, 520.0, np.array([1.0, 4.0 + 0.1j])))
        for _ in range(count):
            i = inc[len(ms)]
            ms.append(tdda.DDAModel(cores[-1], i.nK, i.E0, i.nE0, np.repeat(rng.random(R.size // 3), 3)))
    tdda.solve_multi(ms, 400, 1e-9)
    together = [m.get_P() for m in ms]
    for m, P in zip(ms, together):
        m.InitializeP()
        m.solve_mixed(400, 1e-9)
        assert np.array_equal(m.get_P(), P)
    for m in ms:
        m.close()
    for c in cores:
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("box", [(40, 28, 12), (40, 32, 32), (40, 96, 10), (40, 64, 16), (40, 40, 24), (40, 48, 20)])
def test_paired_plane_blocks_equal_alone(box):
    """Batches of more than two planes an SM run the plane kernel with two blocks an SM (80 x 4
    planes here), a right-hand side alone with one: bit by bit the same."""
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    rng = np.random.Generator(np.random.PCG64(sum(box)))
    R = lattice.bulk(*box)
    core = tdda.AProductCore(*box, R, 10.0, 520.0, np.array([1.0, 2.25 + 0.05j]), max_rhs=4)
    inc = list(lattice.config(3).incidences)[:4]
    rho = np.repeat(0.4 + 0.2 * rng.random(R.size // 3), 3)
    ms = [tdda.DDAModel(core, i.nK, i.E0, i.nE0, rho) for i in inc]
    tdda.solve_batch(ms, tdda.FP32_REFINE, 60, 1e-6)
    batch = [m.get_P() for m in ms]
    for m, P in zip(ms, batch):
        m.InitializeP()
        tdda.solve_batch([m], tdda.FP32_REFINE, 60, 1e-6)
        assert np.array_equal(m.get_P(), P)
    for m in ms:
        m.close()
    core.close()
