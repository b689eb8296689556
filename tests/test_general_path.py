"""The general path's merged kernels against the oracle, bit for bit (the
file they are in is compiled without contraction): periodic wraps at the
domain's edges and inside it, runs (whose depths are derived from SSH after
the first substep) and barotropic_dynamics with and without the biharmonic
term."""
import numpy as np
import pytest

from inmsom_elfs_b200 import basins
from inmsom_elfs_b200.grid import DEPTHS, MEANS, SCRATCH, STATE, Basin, Bounds, Consts

pytestmark = pytest.mark.gpu


def _basin(ora, nx, ny, px, py, inside, scratch):
    """An island basin wrapped in x and/or y; inside > 0: the significant
    area ends that many points before the domain's interior; scratch: other
    values than zero where the loops leave the scratch arrays alone."""
    rng = np.random.default_rng(nx + 3 * px + 5 * py + inside)
    s = Bounds.serial(nx, ny, periodicity_x=px, periodicity_y=py)
    bd = Bounds(*s.astuple()[:8], s.mmm + inside * px, s.mm - inside * px, s.nnn + inside * py, s.nn - inside * py, px, py)
    b = Basin(bd, Consts())
    lu = np.ones(bd.shape, dtype=np.float32, order="F")
    if not py:
        lu[:, :2] = 0.0
        lu[:, -2:] = 0.0
    if not px:
        lu[:2] = 0.0
        lu[-2:] = 0.0
    lu[nx // 3:nx // 3 + 2, ny // 3:ny // 3 + 3] = 0.0
    lu[-4:, ny // 2] = 0.0                        # land at a wrap's source and target
    b.masks["lu"] = np.asfortranarray(lu)
    basins.uniform_metrics(b, 5.0e3)
    for k in b.metrics:                           # metrics that vary in x and y
        b.metrics[k] = np.asfortranarray(b.metrics[k] * (1.0 + 0.05 * rng.random(bd.shape)))
    b.rlh_s = np.asfortranarray(1.0e-4 + 1.0e-5 * rng.standard_normal(bd.shape))
    b.hhq_rest = np.asfortranarray(np.where(lu > 0.5, 200.0 * (0.8 + 0.4 * rng.random(bd.shape)), 0.0))
    b.taux = np.asfortranarray(0.1 * rng.standard_normal(bd.shape))
    b.tauy = np.asfortranarray(0.1 * rng.standard_normal(bd.shape))
    b.forcing["mu"] = np.asfortranarray(300.0 * (1.0 + rng.random(bd.shape)))
    b.forcing["mu4"] = np.full(bd.shape, 1.0e4, order="F")
    b.forcing["rdis"] = np.asfortranarray(1.0e-6 * rng.random(bd.shape))
    b.forcing["wflux"] = np.asfortranarray(1.0e-2 * rng.standard_normal(bd.shape))
    b.dt = 20.0
    b.fill_defaults()
    for k in STATE:
        b.state[k] = np.asfortranarray(0.01 * rng.standard_normal(bd.shape))
    for k in SCRATCH if scratch else ():
        b.scratch[k] = np.asfortranarray(rng.standard_normal(bd.shape))
    basins.finalize(b, ora.OracleBackend())
    ora.hh_init_external(b)
    return b


# sizes: a few blocks of the kernels' 32 x 4 points and ragged edges of them
@pytest.mark.parametrize("nx,ny", [(31, 9), (65, 30)])
@pytest.mark.parametrize("px,py,inside", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (1, 0, 2), (1, 1, 3)])
@pytest.mark.parametrize("what", ["run", "call", "biharmonic"])
def test_general_path_bitexact(gpu, ora, nx, ny, px, py, inside, what):
    # a run reads no scratch array of the host's: the device's start at zero
    b = _basin(ora, nx, ny, px, py, inside, what != "run")
    bo, bg = b.copy(), b.copy()
    with gpu.BarotropicSolver(bg, resident=True, force_general=True) as s:
        if what == "run":
            s.load_state()
            for n in (1, 4):
                ora.run_substeps(bo, n, b.dt)
                s.run_substeps(n, b.dt)
        else:
            ksw4 = int(what == "biharmonic")
            for _ in range(2):
                ora.barotropic_dynamics(bo, 3 * b.dt, 3, ksw4)
                s.barotropic_dynamics(3 * b.dt, 3, ksw4)
        s.sync_to_host(0x1 | 0x2 | (0 if what == "run" else 0x4))
    groups = [("state", STATE), ("depths", DEPTHS)]
    if what != "run":
        groups += [("means", MEANS), ("scratch", SCRATCH)]
    for grp, names in groups:
        for k in names:
            x, y = getattr(bo, grp)[k], getattr(bg, grp)[k]
            assert np.isfinite(x).all() and np.array_equal(x, y), (grp, k, float(np.abs(x - y).max()))
