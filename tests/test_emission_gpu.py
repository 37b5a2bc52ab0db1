"""Furman emission over the whole range of secondary counts, against the oracle
on the same injected uniforms.

The kernel sorts a chunk's secondaries by (count, slot) and inverts with
tabulated constants; the rows here give every count from 0 to 10, so every
starting-guess branch of the inverse incomplete beta runs, and their numbers
straddle the chunk sizes.  Tolerance: the inverses stop at a relative change of
1e-6 of a third-order iteration, which leaves rounding only; 1e-10 of a
velocity is the bound of the replay test of the ordinary yields."""
import numpy as np
import pytest

from conftest import rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu
ME, QE = 9.10938291e-31, 1.602176565e-19


def _rows(n, seed):
    """Absorbed rows on a 20 mm circle with inward normals, 1 to 2000 eV."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0, 2 * np.pi, n)
    nv = -np.stack([np.cos(a), np.sin(a)], 1)
    v = np.sqrt(2 * QE / ME * 10 ** rng.uniform(0, 3.3, n))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    out = np.sum(d[:, :2] * nv, 1) > 0  # towards the wall
    d[out, :2] *= -1
    rows = np.concatenate([-0.02 * nv, d * v[:, None], np.full((n, 1), 1e5)], 1)
    return rows, np.ascontiguousarray(nv)


@pytest.mark.parametrize("n", [1, 31, 33, 1024, 1025, 20001])
@pytest.mark.parametrize("material,sey", [("copper", 1.6), ("copper", 6.0), ("stainless", 9.0)])
def test_all_secondary_counts_match_oracle(gpu, material, sey, n):
    import torch
    from openecloud_b200.grid import Grid
    from openecloud_b200.particleBoundary import AbsorbElliptical
    from openecloud_b200.particleEmitter import FurmanEmitter
    from openecloud_b200.particles import Particles
    rows, nv = _rows(n, 40 + n)
    g = Grid(64, 64, 0.04, 0.04, 1)
    P = Particles("electrons", "variableWeight")
    P.setParticleData(np.zeros((0, 6)))
    P._bind(g)
    bd = AbsorbElliptical(g, P)
    bd.ensure_buffers(n)
    bd._rows[:n] = torch.as_tensor(rows, device="cuda")
    bd._normals[:n] = torch.as_tensor(nv, device="cuda")
    bd._n_abs.fill_(n)
    bd._index = None
    bd._wall_done = True
    bd.absorbedMacroParticleCount = n
    em = FurmanEmitter(bd, P, material=material, seyMax=sey, seed=7)
    u = np.random.default_rng(n).random((n, 32))
    sec = em.generateSecondaries(replay=torch.as_tensor(u, device="cuda")).cpu().numpy()
    ref = O.furman_emit(O.furman(material, sey, None), rows, nv, mode=1, uniforms=u)
    assert sec.shape == ref.shape
    if len(ref):
        assert np.array_equal(sec[:, [0, 1, 5]], ref[:, [0, 1, 5]])
        assert rel_err(sec[:, 2:5], ref[:, 2:5]) <= 1e-10
        assert np.max(np.abs(sec[:, 2:5] - ref[:, 2:5])) <= 1e-10 * np.max(np.abs(ref[:, 2:5]))
    if n > 20000 and material == "copper" and sey > 5:
        assert len(sec) > 60000  # many counts above one


@pytest.mark.parametrize("shift", [8, 16, 24])
def test_work_area_at_any_eight_bytes(gpu, shift):
    """A work area of the stated size that starts at any multiple of 8 bytes gives the
    rows of one from the allocator, and nothing behind its end is written."""
    import torch
    from openecloud_b200.grid import Grid
    from openecloud_b200.particleBoundary import AbsorbElliptical
    from openecloud_b200.particleEmitter import FurmanEmitter
    from openecloud_b200.particles import Particles
    n = 1025
    rows, nv = _rows(n, 5)
    P = Particles("electrons", "variableWeight")
    P.setParticleData(np.zeros((0, 6)))
    g = Grid(64, 64, 0.04, 0.04, 1)
    P._bind(g)
    bd = AbsorbElliptical(g, P)
    bd.ensure_buffers(n)
    bd._rows[:n] = torch.as_tensor(rows, device="cuda")
    bd._normals[:n] = torch.as_tensor(nv, device="cuda")
    bd._n_abs.fill_(n)
    bd._index = None
    bd._wall_done = True
    bd.absorbedMacroParticleCount = n
    em = FurmanEmitter(bd, P, seyMax=6.0, seed=7)
    u = torch.as_tensor(np.random.default_rng(n).random((n, 32)), device="cuda")
    want = em.generateSecondaries(replay=u).clone()
    size = em._work.shape[0]
    area = torch.full((size + 64,), 0x5a, dtype=torch.uint8, device="cuda")
    em._work = area[shift:shift + size]
    em._out.fill_(0.0)
    got = em.generateSecondaries(replay=u)
    assert len(want) > n and torch.equal(got, want)
    assert bool((area[:shift] == 0x5a).all()) and bool((area[shift + size:] == 0x5a).all())


def test_second_chunks_match_oracle(gpu):
    """More rows than all CTAs take as their first chunk (2 x 148 x 1024): the places of a
    second chunk's secondaries follow from the sums of the rows between."""
    test_all_secondary_counts_match_oracle(gpu, "copper", 1.6, 320_001)
