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


# box, right-hand sides: the number of branches of a solve's steps there on 152 SMs
BRANCHES = [((20, 20, 10), 3, 1), ((48, 6, 6), 2, 2), ((48, 6, 6), 7, 2), ((48, 6, 6), 3, 3), ((20, 20, 10), 5, 2),
            ((20, 20, 10), 8, 2), ((20, 24, 20), 5, 4), ((33, 24, 12), 4, 4)]


def _core(box, n):
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    R = lattice.bulk(*box)
    return tdda.AProductCore(*box, R, 10.0, 520.0, MAT, max_rhs=n), R


@pytest.mark.gpu
@pytest.mark.parametrize("loop", ["1", "0"])
@pytest.mark.parametrize("box,n,branches", BRANCHES)
def test_batch_tuner_times_the_branches_of_a_solve(box, n, branches, loop, monkeypatch):
    """The candidates are timed on solver steps, the whole batch in its branches: by the kernels that
    eight more steps of each launch, in two rounds (24 products asked for, and 8)."""
    monkeypatch.setenv("TDDA_DEVICE_LOOP", loop)
    core, _ = _core(box, n)

    def tune(reps):
        before = tdda.kernel_launches()
        t = core.autotune_batch(nrhs=n, reps=reps)
        assert t["group"] == min(t["candidates"], key=lambda k: k["ms"])["group"]
        assert all(k["ms"] > 0 for k in t["candidates"])
        return tdda.kernel_launches() - before, [k["group"] for k in t["candidates"]]

    tune(8)
    (few, groups), (many, _) = tune(8), tune(24)
    sets = [branches if g == 0 else -(-n // g) for g in groups]
    ends = 2  # the step end after every fourth step
    assert groups[0] == 0
    assert many - few == 2 * (16 * core.pass_count(tdda.FP32_REFINE) * sum(sets) + ends * len(groups))
    core.close()


@pytest.mark.gpu
@pytest.mark.parametrize("box,n,branches", [((20, 20, 10), 1, 1), ((48, 6, 6), 3, 3), ((20, 24, 20), 5, 4), ((97, 12, 9), 2, 2)])
def test_x_tuner_times_solver_steps(box, n, branches):
    """The gather's tiles and the forms likewise: tiles tie on plain products and not in a step."""
    core, _ = _core(box, n)

    def tune(reps):
        before = tdda.kernel_launches()
        t = core.autotune(nrhs=n, reps=reps)
        best = min(t["candidates"], key=lambda k: k["ms"])
        assert (t["x_form"], t["x_tile"]) == (best["form"], best["tile"]) and best["ms"] > 0
        return tdda.kernel_launches() - before, [(k["form"], k["tile"]) for k in t["candidates"]]

    tune(8)
    (few, cands), (many, _) = tune(8), tune(24)
    want = 0
    for form, tile in cands:
        core.set_xpass(form, tile)
        x_first = core.pass_names(tdda.FP32_REFINE)[0] == "k_xfwd"  # the z-y-x passes take no branches
        want += 2 * (16 * core.pass_count(tdda.FP32_REFINE) * (branches if x_first else 1) + 2)
    assert many - few == want
    core.close()


@pytest.mark.gpu
def test_tuners_of_a_core_of_one_material():
    """Such a core has no models; its products are timed."""
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    c = tdda.AProductCore(9, 8, 7, lattice.bulk(9, 8, 7), 10.0, 520.0, MAT[:1], max_rhs=2)
    t = c.autotune_batch(nrhs=2, reps=2)
    assert [k["group"] for k in t["candidates"]] == [0, 1] and all(k["ms"] > 0 for k in t["candidates"])
    t = c.autotune(nrhs=2, reps=2)
    assert all(k["ms"] > 0 for k in t["candidates"])
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("box,n,branches", BRANCHES)
def test_solves_run_in_their_branches(box, n, branches, monkeypatch):
    """The number of branches of a solve's steps: the kernels that eight more steps launch, beside
    those of eight more steps with a launch for each right-hand side."""
    monkeypatch.setenv("TDDA_DEVICE_LOOP", "0")
    core, R = _core(box, n)
    rng = np.random.Generator(np.random.PCG64(n))
    inc = (list(lattice.config(3).incidences) * 2)[:n]
    ms = [tdda.DDAModel(core, i.nK, i.E0, i.nE0, np.repeat(rng.random(R.size // 3), 3)) for i in inc]
    tdda.solve_batch(ms, tdda.FP32_REFINE, 4, 1e-30)  # what a core and its models make once

    def launched(steps):
        for m in ms:
            m.InitializeP()
        before = tdda.kernel_launches()
        tdda.solve_batch(ms, tdda.FP32_REFINE, steps, 1e-30)
        return tdda.kernel_launches() - before

    more = {}
    for group in (0, 1):
        core.set_batch_group(group)
        more[group] = launched(12) - launched(4)
    ends = 2  # the step end after every fourth step
    assert more[1] == 16 * core.pass_count(tdda.FP32_REFINE) * n + ends
    assert more[0] == 16 * core.pass_count(tdda.FP32_REFINE) * branches + ends
    for m in ms:
        m.close()
    core.close()


@pytest.mark.gpu
@pytest.mark.parametrize("loop", ["1", "0"])
@pytest.mark.parametrize("box,n", [((20, 24, 20), 5), ((33, 24, 12), 4), ((25, 26, 11), 6)])
def test_four_branches_equal_alone(box, n, loop, monkeypatch):
    """Four branches, of equal and unequal shares: each solution bit by bit the one solved alone."""
    monkeypatch.setenv("TDDA_DEVICE_LOOP", loop)
    core, R = _core(box, n)
    rng = np.random.Generator(np.random.PCG64(sum(box)))
    inc = (list(lattice.config(3).incidences) * 2)[:n]
    ms = [tdda.DDAModel(core, i.nK, i.E0, i.nE0, np.repeat(rng.random(R.size // 3), 3)) for i in inc]
    infos = tdda.solve_batch(ms, tdda.FP32_REFINE, 400, 1e-8)
    batch = [m.get_P() for m in ms]
    for k, m in enumerate(ms):
        m.InitializeP()
        [alone] = tdda.solve_batch([m], tdda.FP32_REFINE, 400, 1e-8)
        assert alone["inner_iterations"] == infos[k]["inner_iterations"]
        assert np.array_equal(m.get_P(), batch[k])
    for m in ms:
        m.close()
    core.close()
