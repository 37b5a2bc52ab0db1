"""sortByColumn at the edges of its 4096-key tiles and of the digit scan, against
a stable host argsort of the stored values: exact for every field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("col", [2, 4, 5, 6])
@pytest.mark.parametrize("n", [1, 2, 33, 4095, 4096, 4097, 12_289])
def test_sort_is_stable_at_tile_edges(gpu, n, col):
    from openecloud_b200.grid import Grid
    from openecloud_b200.particles import Particles
    rng = np.random.default_rng(n + col)
    g = Grid(70, 90, 0.04, 0.04, 0)
    pd = np.empty((n, 6))
    pd[:, 0:2] = rng.uniform(-0.0199, 0.0199, (n, 2))
    pd[:, 2:5] = rng.choice([-2e6, -1.5, -0.0, 0.0, 3.0, 1e6], (n, 3))  # signs, zeros and many equal keys
    pd[:, 5] = rng.choice([0.25, 1.0, 1.0 + 2 ** -20, 7e8], n)
    P = Particles("electrons", "variableWeight")
    P.setParticleData(pd)
    P._bind(g)
    soa = {k: v[:n].cpu().numpy().copy() for k, v in P.soa().items()}
    key = soa[{2: "vx", 4: "vz", 5: "w", 6: "cell"}[col]]
    if col != 6:  # the order of the float bits: -0 before +0
        u = key.view(np.uint32)
        key = np.where(u >> 31, ~u, u | 0x80000000).astype(np.uint32)
    order = np.argsort(key, kind="stable")
    P.sortByColumn(col)
    for k, v in P.soa().items():
        assert np.array_equal(v[:n].cpu().numpy().view(np.uint32), soa[k][order].view(np.uint32)), k


@pytest.mark.parametrize("n", [1, 4097, 12_289])
def test_cell_sort_stays_in_its_work_area(gpu, n):
    """oec_cell_sort_work_bytes suffices for a sort by cell: what lies behind is untouched."""
    import torch
    from openecloud_b200 import _lib
    from openecloud_b200 import device as D
    from openecloud_b200.grid import Grid
    from openecloud_b200.particles import Particles
    rng = np.random.default_rng(n)
    P = Particles("electrons", "variableWeight")
    pd = np.ones((n, 6))
    pd[:, 0:2] = rng.uniform(-0.0199, 0.0199, (n, 2))
    P.setParticleData(pd)
    P._bind(Grid(70, 90, 0.04, 0.04, 0))
    cell = P.soa()["cell"][:n].cpu().numpy()
    size = int(_lib.lib().oec_cell_sort_work_bytes(P._cap))
    area = torch.full((size + 4096,), 0x5a, dtype=torch.uint8, device="cuda")
    tmp = P.c_scratch()
    _lib.call("oec_sort_particles", P.c_particles(), tmp, 6, area.data_ptr(), D.stream())
    assert bool((area[size:] == 0x5a).all())
    assert np.array_equal(P._sort_tmp["cell"][:n].cpu().numpy(), np.sort(cell))
