"""The kernels with one result per dipole, design parameter or observation point (al, internal
field, density gradient, off-lattice field) at the edges of their blocks, against the host's
64-bit formulas.  Tolerances: al and the internal field are some 20 rounded operations each
(20 x 1.1e-16 < 1e-14); a sum of n terms is within n x 1.1e-16 of the terms' magnitudes
(n <= 3 x 600 here: 2e-13, and the terms themselves 1e-14: 1e-12)."""
import math

import numpy as np
import pytest

import oracle as O
import tdda
from conftest import rel
from tdda import topo

pytestmark = pytest.mark.gpu
D, LAM = 9.0, 520.0
K = 2 * math.pi / LAM
NK, NE0 = np.array([0.0, math.sin(0.4), math.cos(0.4)]), np.array([0.0, math.cos(0.4), -math.sin(0.4)])


def _setup(box, material):
    if tdda.device_count() < 1:
        pytest.skip("no CUDA device")
    R = np.array([(x, y, z) for x in range(box[0]) for y in range(box[1]) for z in range(box[2])], np.int32).ravel()
    rng = np.random.Generator(np.random.PCG64(sum(box)))
    rho = np.repeat(0.05 + 0.9 * rng.random(R.size // 3), 3)
    core = tdda.AProductCore(*box, R, D, LAM, np.array(material), 1.0)
    m = tdda.DDAModel(core, NK, 1.0, NE0, rho)
    P = rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size)
    m.InitializeP(P)
    return core, m, R, rho, P, rng


@pytest.mark.parametrize("box", [(2, 1, 1), (43, 3, 1), (32, 4, 1)])  # 2, 129 and 128 dipoles
@pytest.mark.parametrize("eps2", [2.25 + 0j, -12.5 + 0.8j, -2.1 + 3.9j])
def test_al_over_materials(box, eps2):
    core, m, R, rho, P, rng = _setup(box, [1.0 + 0.02j, eps2])
    m0, m1 = core.material  # the table as the core normalises it
    eps = m0 + rho * (m1 - m0)
    al = np.array([1.0 / O.get_alpha(LAM, K, D, e, NE0, NK) for e in eps])
    assert rel(m.get_al(), al) <= 1e-14
    m.close()


@pytest.mark.parametrize("nparam", [1, 32, 33, 70])
def test_gradient_lists_longer_than_a_chunk(nparam):
    core, m, R, rho, P, rng = _setup((7, 6, 5), [1.0 + 0.02j, 5.0 + 0.3j])
    adj = [tdda.DDAModel(core, NK, 1.0, NE0, rho) for _ in range(2)]
    lam = [rng.standard_normal(R.size) + 1j * rng.standard_normal(R.size) for _ in adj]
    for a, v in zip(adj, lam):
        a.InitializeP(v)
    sizes = np.array(([600, 0, 1, 255, 256, 257, 3] * 10)[:nparam])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    dip = rng.integers(0, R.size // 3, off[-1]).astype(np.int32)
    coef = np.array([0.3 - 0.8j, 1.1 + 0.2j])
    got = m.density_gradient(adj, coef, off, dip)
    step = core.material[1] - core.material[0]
    eps = core.material[0] + rho * step
    S = float(np.sum((NE0 * NK) ** 2))
    term = np.real((coef[0] * lam[0] + coef[1] * lam[1]) * topo.dal_deps(eps, K, D, S) * step * P).reshape(-1, 3)
    for i in range(nparam):
        t = term[dip[off[i]:off[i + 1]]]
        assert abs(got[i] - math.fsum(t.ravel())) <= 1e-12 * np.abs(t).sum() * 4, i
    for a in adj + [m]:
        a.close()


@pytest.mark.parametrize("box,npts", [((3, 2, 2), 1), ((3, 2, 2), 5), ((24, 20, 18), 1), ((24, 20, 18), 9)])
def test_field_over_one_and_many_partials(box, npts):
    core, m, R, rho, P, rng = _setup(box, [1.0 + 0.02j, 5.0 + 0.3j])
    pts = D * np.array(box) + rng.uniform(5.0, 200.0, (npts, 3))
    got = m.field_at(pts)
    Rd = D * R.reshape(-1, 3)
    for p, g in zip(pts, got):
        t = topo.ldr_tensor(K, *(p[:, None] - Rd.T))
        xx, xy, xz, yy, yz, zz = t
        q = P.reshape(-1, 3).T
        f = np.array([xx * q[0] + xy * q[1] + xz * q[2], xy * q[0] + yy * q[1] + yz * q[2],
                      xz * q[0] + yz * q[1] + zz * q[2]])
        want = NE0 * np.exp(1j * K * (NK @ p)) - f.sum(axis=1)
        assert np.max(np.abs(g - want)) <= 1e-12 * (1 + np.abs(f).sum())
    m.close()
