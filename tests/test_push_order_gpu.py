"""The fused step on stores in cell order and in random order.

A CTA decides from its first chunk whether its particles are near each other
(windows in shared memory) or not (pairs of lanes straight to the grid).  Both
give the same particles and the same integer deposit, so a random order and
the cell order of the same rows must agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step(rows, bound, btype):
    import torch
    from openecloud_b200.grid import Grid
    from openecloud_b200.particleBoundary import AbsorbElliptical, AbsorbRectangular
    from openecloud_b200.particles import Particles
    g = Grid(150, 220, 0.04, 0.06, bound)
    P = Particles("electrons", "variableWeight")
    P.setBConst([0.0, 0.5, 0.0])
    P.setParticleData(rows)
    P._bind(g)
    G = g.getNpExt()
    e = P.fieldTable(g, np.random.default_rng(1).normal(0, 1e4, 2 * G), 2)
    b = P.fieldTable(g, np.random.default_rng(2).normal(0, 0.1, 3 * G), 3) if btype == 2 else None
    bd = (AbsorbRectangular if bound == 0 else AbsorbElliptical)(g, P)
    P.pushGatherDeposit(g, e, 3e-11, btype, bd, bCellTable=b)
    torch.cuda.synchronize()
    fix, scale = P.getChargeOnGridFixed()
    return P.getParticleData(), P.getIsInside(), fix, scale


@pytest.mark.parametrize("bound,btype", [(0, 0), (1, 1), (1, 2)])
@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 2047, 50_001])
def test_random_and_cell_order_agree(gpu, n, bound, btype):
    rng = np.random.default_rng(n)
    rows = np.empty((n, 6))
    rows[:, 0], rows[:, 1] = rng.uniform(-0.0199, 0.0199, n), rng.uniform(-0.0299, 0.0299, n)
    rows[:, 2:5] = rng.normal(0, 2e6, (n, 3))
    rows[:, 5] = rng.uniform(0.5, 2.0, n)
    order = np.lexsort((rows[:, 0], np.floor(rows[:, 1] / (0.06 / 219))))
    a, ina, fa, sa = _step(rows, bound, btype)
    b, inb, fb, sb = _step(rows[order], bound, btype)
    assert sa == sb and np.array_equal(fa, fb)
    assert np.array_equal(a[order], b) and np.array_equal(ina[order], inb)
    # the deposit is exact: every survivor's whole quantised charge is on the grid
    assert fa.sum() == np.rint(rows[ina == 1, 5].astype(np.float32).astype(np.float64) * sa).sum()


@pytest.mark.parametrize("bound,btype", [(0, 0), (1, 1), (1, 2)])
def test_empty_store(gpu, bound, btype):
    """A store without particles (every one was removed): nothing is read, absorbed or
    deposited, and what lies in the arrays stays as it was."""
    import torch
    from openecloud_b200.grid import Grid
    from openecloud_b200.particleBoundary import AbsorbElliptical, AbsorbRectangular
    from openecloud_b200.particles import Particles
    g = Grid(40, 30, 0.04, 0.06, bound)
    P = Particles("electrons", "variableWeight")
    P.setParticleData(np.tile([0.001, 0.002, 1e5, 2e5, 3e5, 1.0], (2000, 1)))
    P._bind(g)
    P.setMacroParticleCount(0)
    P._deposit_buffers(g)
    P._rho_fix.fill_(7)
    P._status.fill_(0)
    before = {k: v.clone() for k, v in P.soa().items()}
    e = P.fieldTable(g, np.ones(2 * g.getNpExt()), 2)
    b = P.fieldTable(g, np.ones(3 * g.getNpExt()), 3) if btype == 2 else None
    bd = (AbsorbRectangular if bound == 0 else AbsorbElliptical)(g, P)
    for _ in range(2):
        P.pushGatherDeposit(g, e, 3e-11, btype, bd, bCellTable=b)
    torch.cuda.synchronize()
    assert P.getMacroParticleCount() == 0 and not P._rho_fix.any()
    assert all(torch.equal(P.soa()[k], before[k]) for k in before)
    assert not any(P.status().values())


@pytest.mark.parametrize("rows_apart", [7, 8, 9])
def test_chunks_at_the_limit_of_the_deposit_choice(gpu, rows_apart):
    """Chunks whose first and last particle lie 8 rows apart, the limit up to which a CTA
    takes the windows, and whose particles cross many rows in the push, so that a choice
    made again from moved cells would come out differently: every launch deposits what
    the same particles deposit in random order."""
    import torch
    from openecloud_b200.grid import Grid
    from openecloud_b200.particleBoundary import AbsorbRectangular
    from openecloud_b200.particles import Particles
    g = Grid(64, 96, 0.04, 0.06, 0)
    dx, dy, n = g.getDx(), g.getDy(), 40 * 1024
    rng = np.random.default_rng(rows_apart)
    k, chunk = np.arange(n) % 1024, np.arange(n) // 1024
    cell_y = 30 + chunk % 20 + np.rint(k * rows_apart / 1023.0)
    rows = np.empty((n, 6))
    rows[:, 0] = (20 + rng.integers(0, 3, n) + rng.uniform(0.1, 0.9, n)) * dx - 0.02
    rows[:, 1] = (cell_y + rng.uniform(0.1, 0.9, n)) * dy - 0.03
    rows[:, 2], rows[:, 4] = rng.normal(0, 1e6, n), 0.0
    rows[:, 3] = rng.uniform(-12, 12, n) * dy / 3e-11
    rows[:, 5] = rng.uniform(0.5, 2.0, n)
    e = np.zeros(2 * g.getNpExt())

    def step(r):
        P = Particles("electrons", "variableWeight")
        P.setBConst([0.0, 0.1, 0.0])
        P._bind(g)
        out = []
        for _ in range(30):
            P.setParticleData(r)
            P.pushGatherDeposit(g, P.fieldTable(g, e, 2), 3e-11, 1, AbsorbRectangular(g, P))
            out.append(P._rho_fix.clone())
        torch.cuda.synchronize()
        return out

    got, want = step(rows), step(rows[rng.permutation(n)])
    assert want[0].any() and all(torch.equal(x, want[0]) for x in got + want)


@pytest.mark.parametrize("bound,btype", [(0, 0), (1, 1)])
def test_several_chunks_per_cta(gpu, bound, btype):
    """More chunks than resident CTAs (four on each of 148 SMs), in random and in cell order."""
    test_random_and_cell_order_agree(gpu, 700_001, bound, btype)


@pytest.mark.parametrize("btype", [0, 2])
@pytest.mark.parametrize("n", [1025, 500_001])
def test_cut_cells_and_uneven_weights(gpu, n, btype):
    """The cut-cell wall (three CTAs per SM, 500,001 electrons are more chunks than those)
    with weights from 1e-9 to 1, so that charges lie on both sides of the 2^40 up to which
    the windows take them without a test: both orders agree and the deposit is exact."""
    import torch
    from openecloud_b200.grid import Grid
    from openecloud_b200.particleBoundary import AbsorbArbitraryCutCell
    from openecloud_b200.particles import Particles
    rng = np.random.default_rng(n)
    rows = np.empty((n, 6))
    rows[:, 0], rows[:, 1] = rng.uniform(-0.0199, 0.0199, n), rng.uniform(-0.0299, 0.0299, n)
    rows[:, 2:5] = rng.normal(0, 2e6, (n, 3))
    rows[:, 5] = 10 ** rng.uniform(-9, 0, n)
    order = np.lexsort((rows[:, 0], np.floor(rows[:, 1] / (0.06 / 219))))
    g = Grid(150, 220, 0.04, 0.06, 1)
    e = np.random.default_rng(1).normal(0, 1e4, 2 * g.getNpExt())
    b = np.random.default_rng(2).normal(0, 0.1, 3 * g.getNpExt())
    got = []
    for r in (rows, rows[order]):
        P = Particles("electrons", "variableWeight")
        P.setParticleData(r)
        P._bind(g)
        tabs = P.fieldTable(g, e, 2), P.fieldTable(g, b, 3) if btype == 2 else None
        P.pushGatherDeposit(g, tabs[0], 3e-11, btype, AbsorbArbitraryCutCell(g, P), bCellTable=tabs[1])
        torch.cuda.synchronize()
        got.append((P.getParticleData(), P.getIsInside(), *P.getChargeOnGridFixed()))
    (pa, ina, fa, sa), (pb, inb, fb, sb) = got
    assert sa == sb and np.array_equal(fa, fb) and 0 < ina.sum() < n
    assert np.array_equal(pa[order], pb) and np.array_equal(ina[order], inb)
    q = np.rint(rows[ina == 1, 5].astype(np.float32).astype(np.float64) * sa)
    assert q.min() < 2.0 ** 40 < q.max() and int(fa.sum()) == sum(int(x) for x in q)
