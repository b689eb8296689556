"""Copies between host arrays and the device's pitched rows: rows below
8 KB travel packed (a kernel moves them into the pitched rows), longer ones
pitched.  Sizes on both sides of that line, for 8-byte fields (1024 columns)
and 4-byte masks (2048), odd and even, one level and several; every point of
an array, its border included."""
import numpy as np
import pytest

from inmsom_elfs_b200 import basins
from test_baroclinic import TAU, _gpu_run, _run_oracle, coastline, inputs
from test_tracer import inputs as tracer_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(5, 4), (333, 9), (1019, 6), (1020, 6), (1021, 5), (2043, 3), (2044, 3)])
@pytest.mark.parametrize("nz", [1, 3])
def test_fields_keep_every_point(gpu, ora, nx, ny, nz):
    b = basins.beta_plane_basin(n=nx, ny=ny, seed=nx + nz)
    basins.finalize(b, ora.OracleBackend())
    rng = np.random.default_rng(nx * nz)
    dz = rng.random(nz)
    u = np.asfortranarray(rng.standard_normal((*b.bounds.shape, nz)))
    utr = np.asfortranarray(rng.standard_normal(b.bounds.shape))
    mask = np.asfortranarray((rng.random(b.bounds.shape) > 0.4).astype(np.float32))
    wu, wt = u.copy(order="F"), utr.copy(order="F")
    s = np.zeros(b.bounds.shape)
    for k in range(nz):
        s = s + u[..., k] * dz[k]
    on = mask > 0.5
    on[[0, -1]] = on[:, [0, -1]] = False
    wt[on] = s[on]
    for k in range(nz):
        wu[..., k][on] = u[..., k][on] - s[on]
    with gpu.BarotropicSolver(b) as sol:
        sol.depth_ave(dz, u, utr, mask, 1)
        for k, v in b.state.items():
            v[...] = rng.standard_normal(v.shape)
        want = {k: v.copy() for k, v in b.state.items()}
        sol.load_state()
        for v in b.state.values():
            v[...] = 0.0
        sol.sync_to_host()
    assert np.array_equal(u, wu) and np.array_equal(utr, wt)
    for k, v in want.items():
        assert np.array_equal(b.state[k], v), k


@pytest.mark.parametrize("nx,ny,nz", [(1019, 12, 3), (1021, 9, 4), (40, 3, 5), (33, 30, 2)])
def test_banded_calls_bitexact(gpu, ora, nx, ny, nz):
    """The 3-D calls' row bands (fewer rows than bands among them)."""
    b = coastline(ora, nx=nx, ny=ny, seed=nz)
    dz, hzt, f = inputs(b, nz=nz, seed=nz)
    got, _ = _gpu_run(gpu, b, dz, hzt, f)
    for g, w in zip(got, _run_oracle(ora, b, dz, hzt, f)):
        assert np.array_equal(g, w)
    dz, hzt, f = tracer_inputs(b, nz=nz, seed=nz)
    fl = [np.asfortranarray(np.random.default_rng(k).standard_normal((*b.bounds.shape, 4))) for k in (1, 2)]
    st = [f["ff"].copy(order="F"), f["ffp"].copy(order="F"), *[x.copy(order="F") for x in fl]]
    with gpu.BarotropicSolver(b) as s:
        s.tracer_tran_diff(dz, hzt, TAU, *st, f)
    want = [f["ff"].copy(order="F"), f["ffp"].copy(order="F"), *[x.copy(order="F") for x in fl]]
    ora.tracer_tran_diff(b, dz, hzt, TAU, *want, f)
    for g, w in zip(st, want):
        assert np.array_equal(g, w)
