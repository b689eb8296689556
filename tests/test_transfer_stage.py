"""The device buffer that packed uploads go through: its size is bounded,
whatever the fields' size, and fields larger than it go through it in runs of
levels, or of a level's rows.  A device without the memory for it (here: a
limit below one row) takes the pitched copies, as do rows that are a multiple
of 128 bytes and every download."""
import ctypes

import numpy as np
import pytest
from conftest import rel_err

from inmsom_elfs_b200 import _lib, basins
from test_baroclinic import TAU, _run_oracle, coastline, inputs

pytestmark = pytest.mark.gpu


def _depth_ave(b, sol, nz, seed):
    """One call on nz levels (3 fields in, 2 out) against numpy, bit for bit."""
    rng = np.random.default_rng(seed)
    dz = rng.random(nz)
    u = np.asfortranarray(rng.standard_normal((*b.bounds.shape, nz)))
    utr = np.asfortranarray(rng.standard_normal(b.bounds.shape))
    mask = np.asfortranarray((rng.random(b.bounds.shape) > 0.4).astype(np.float32))
    s = np.zeros(b.bounds.shape)
    for k in range(nz):
        s = s + u[..., k] * dz[k]
    on = mask > 0.5
    on[[0, -1]] = on[:, [0, -1]] = False
    wu, wt = u.copy(order="F"), utr.copy(order="F")
    wt[on] = s[on]
    for k in range(nz):
        wu[..., k][on] = u[..., k][on] - s[on]
    sol.depth_ave(dz, u, utr, mask, 1)
    assert np.array_equal(u, wu) and np.array_equal(utr, wt)


def _baroclinic(sol, dz, hzt, f):
    st = [f[k].copy(order="F") for k in ("uu", "uup", "vv", "vvp")]
    return sol.baroclinic_dynamics(dz, hzt, TAU, *st, **{k: f[k] for k in sol.BAROCLINIC_FIELDS})


def test_stage_is_bounded(gpu, ora):
    """A field of 122 MB (504 x 504 x 60) through a buffer of 64 MB: the
    device's free memory falls by no more than that and the driver's own
    bookkeeping (8 MiB)."""
    import torch
    b = coastline(ora, nx=500, ny=500, seed=2)
    with gpu.BarotropicSolver(b) as sol:
        _baroclinic(sol, *inputs(b, nz=60, seed=3))   # takes the levels' block
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info(0)[0]
        _depth_ave(b, sol, 60, 4)
        torch.cuda.synchronize()
        taken = free0 - torch.cuda.mem_get_info(0)[0]
        assert taken <= (64 + 8) << 20, taken / 2**20


# 30 x 20 points: rows of 272 bytes, levels of 6528; stages that hold one row
# (and a little more), part of a level, one level, several, all but one
@pytest.mark.parametrize("limit", [272, 700, 4000, 6528, 20000, 6528 * 5 - 1])
@pytest.mark.parametrize("nx,ny,nz", [(30, 20, 5), (301, 7, 4)])
def test_small_stages(gpu, ora, nx, ny, nz, limit):
    b = coastline(ora, nx=nx, ny=ny, seed=nz)
    limit = max(limit, (nx + 4) * 8)
    with gpu.BarotropicSolver(b) as sol:
        assert _lib.load().inmsom_test_stage_limit(sol._ctx, limit) == _lib.OK
        _depth_ave(b, sol, nz, limit)


@pytest.mark.parametrize("limit", [1 << 12, 1 << 15, 1 << 17])
def test_small_stages_banded(gpu, ora, limit):
    b = coastline(ora, nx=90, ny=40, seed=8)
    dz, hzt, f = inputs(b, nz=6, seed=9)
    want = _run_oracle(ora, b, dz, hzt, f)
    with gpu.BarotropicSolver(b) as sol:
        assert _lib.load().inmsom_test_stage_limit(sol._ctx, limit) == _lib.OK
        got = _baroclinic(sol, dz, hzt, f)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("limit", [0, 1, 271])
def test_no_memory_for_a_stage(gpu, ora, limit):
    b = coastline(ora, nx=30, ny=20, seed=5)
    ora.hh_init_external(b)
    with gpu.BarotropicSolver(b) as sol:
        assert _lib.load().inmsom_test_stage_limit(sol._ctx, limit) == _lib.OK
        _depth_ave(b, sol, 5, limit)
        dz, hzt, f = inputs(b, nz=4, seed=9)
        for g, w in zip(_baroclinic(sol, dz, hzt, f), _run_oracle(ora, b, dz, hzt, f)):
            assert np.array_equal(g, w)
        bo = b.copy()
        sol.barotropic_dynamics(2 * b.dt, 2)
        ora.barotropic_dynamics(bo, 2 * b.dt, 2)
        for k, v in bo.state.items():
            assert rel_err(b.state[k], v) <= 1e-12, k


@pytest.mark.parametrize("nx,ny", [(5, 4), (28, 20), (30, 20), (90, 43), (124, 30), (400, 300)])
def test_stages_are_allocated_once(gpu, ora, nx, ny):
    """One allocation serves every 2-D upload of a context, one the bands of
    a 3-D call (the last band is the tallest); none where rows of 4- and
    8-byte values are multiples of 128 bytes (32 and 128 columns)."""
    b = coastline(ora, nx=nx, ny=ny, seed=5)
    ora.hh_init_external(b)
    once = 0 if (nx + 4) % 32 == 0 else 1

    def allocs():
        n = ctypes.c_int()
        assert _lib.load().inmsom_test_stage_allocs(sol._ctx, ctypes.byref(n)) == _lib.OK
        return n.value

    with gpu.BarotropicSolver(b) as sol:
        assert allocs() == once
        sol.load_state()
        sol.barotropic_dynamics(2 * b.dt, 2, 1)
        assert allocs() == once
        dz, hzt, f = inputs(b, nz=4, seed=9)
        want = _run_oracle(ora, b, dz, hzt, f)
        for _ in range(2):
            for g, w in zip(_baroclinic(sol, dz, hzt, f), want):
                assert np.array_equal(g, w)
            assert allocs() == 2 * once
        _depth_ave(b, sol, 4, nx)


def test_stage_limit_argument_checks():
    assert _lib.load().inmsom_test_stage_limit(None, 0) == _lib.EARG
    assert _lib.load().inmsom_test_stage_allocs(None, None) == _lib.EARG
