"""Work items of the fused path on basins whose strips hold runs of land:
items cover the ocean rows of a strip and land runs of up to eight rows
between them, and are cut down to one row on a small basin.  Against the
oracle after 10 steps; the fused path's tolerance is 1e-12 normwise."""
import numpy as np
import pytest
from conftest import rel_err

from inmsom_elfs_b200 import basins
from inmsom_elfs_b200.grid import STATE


def _banded(ora, nx, ny, bands, seed):
    """A beta-plane basin with land across its rows: bands of (first interior
    row, rows), and one lone ocean row between two of them at the east end."""
    b = basins.beta_plane_basin(n=nx, ny=ny, seed=seed)
    j0 = b.bounds.ny_start - b.bounds.bnd_y1
    for first, rows in bands:
        b.masks["lu"][: 3 * nx // 4, j0 + first:j0 + first + rows] = 0.0
        b.masks["lu"][3 * nx // 4:, j0 + first + 1:j0 + first + rows] = 0.0
    b.hhq_rest[b.masks["lu"] < 0.5] = 0.0
    basins.finalize(b, ora.OracleBackend())
    rng = np.random.default_rng(seed)
    for k in ("ssh_e", "sshp_e"):
        b.state[k] = np.asfortranarray(0.1 * rng.standard_normal(b.bounds.shape) * b.masks["lu"])
    ora.hh_init_external(b)
    return b


# land runs shorter than, at and past the eight rows an item spans; sizes
# from one row per item to several rows, and strips of one or two columns
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,bands", [
    (31, 40, [(3, 1), (9, 7), (20, 8), (31, 5)]),
    (62, 60, [(2, 9), (13, 8), (23, 10), (40, 20)]),
    (400, 170, [(10, 9), (21, 8), (60, 30), (100, 1), (140, 12)]),
    (700, 500, [(1, 40), (60, 9), (200, 8), (300, 100)]),
])
@pytest.mark.parametrize("call", [False, True])
def test_land_runs_in_the_strips(gpu, ora, nx, ny, bands, call):
    b = _banded(ora, nx, ny, bands, seed=nx + ny)
    bo, bg = b.copy(), b.copy()
    with gpu.BarotropicSolver(bg, resident=True) as s:
        assert s.path()[0] == 1
        s.load_state()
        if call:
            ora.barotropic_dynamics(bo, 5 * b.dt, 5)
            s.barotropic_dynamics(5 * b.dt, 5)
        else:
            ora.run_substeps(bo, 10, b.dt)
            s.run_substeps(10, b.dt)
        s.sync_to_host()
    for k in STATE:
        assert rel_err(bg.state[k], bo.state[k]) <= 1e-12, k
        assert np.array_equal(bg.state[k][b.masks["lu"] < 0.5], b.state[k][b.masks["lu"] < 0.5]), k
    if call:
        for k, v in bo.means.items():
            assert rel_err(bg.means[k], v) <= 1e-12, k


# a basin alone of few waves of items takes the ring of four slots, an
# ensemble's member the ring of five: the same values bit for bit (items of
# 1-2 rows, about 7, several waves; past four waves both take five)
@pytest.mark.gpu
@pytest.mark.parametrize("kind,nx,ny", [
    ("beta", 31, 31), ("beta", 330, 330), ("beta", 1300, 1300), ("beta", 1750, 1750),
    ("regional", 300, 200), ("spherical", 45, 33), ("spherical", 701, 487), ("spherical", 1800, 1300),
])
def test_ring_sizes_agree(gpu, ora, kind, nx, ny):
    if kind == "beta":
        b = basins.beta_plane_basin(n=nx, seed=nx)
    elif kind == "regional":
        b = basins.regional_basin(nx=nx, ny=ny, seed=nx)
    else:
        b = basins.spherical_basin(nx=nx, ny=ny, dxst=12.0 / nx, dyst=8.0 / ny, dt=2.0)
    basins.finalize(b, ora.OracleBackend())
    ora.hh_init_external(b)
    b1, b2 = b.copy(), b.copy()
    with gpu.BarotropicSolver(b1, resident=True) as s:
        assert s.path()[0] == 1
        s.load_state()
        s.run_substeps(6, b.dt)
        s.sync_to_host()
    with gpu.BarotropicSolver(b2, resident=True) as s:
        s.load_state()
        with gpu.Ensemble([s], group=2) as e:
            e.run(6, [b.dt], np.ones(6))
        s.sync_to_host()
    for k in STATE:
        assert np.array_equal(b1.state[k], b2.state[k]), k
    assert np.abs(b1.state["ubrtr_e"]).max() > 0.0
