"""The precision form's deposit where a warp's cells hold different counts: spreads on both sides of
64 (the two ways the warp's quota is chosen) and of 32 (one or two passes over the excess), species
of other counts, one of them a single particle, after one another in the same tiles (their buckets
are loaded a species ahead), grids of one tile and of several. Bar: relative L2 error
<= 1e-5 per moment against the FP64 oracle; a particle left out or taken twice is above 1e-4."""
import numpy as np
import pytest

import oracle
from sputnipic_b200 import workload as W
from test_precision_gpu import oracle64, rel_l2, run_sim

pytestmark = pytest.mark.gpu


def at_rest(rng, wl, counts):
    """counts[cell] particles inside each cell, too slow to leave it in a step."""
    cell = np.repeat(np.arange(counts.size), counts.ravel())
    ijk = np.unravel_index(cell, counts.shape)
    p = {k: ((i + rng.uniform(0.1, 0.9, cell.size)) * L / c).astype(np.float32)
         for k, i, L, c in zip("xyz", ijk, (wl.Lx, wl.Ly, wl.Lz), counts.shape)}
    for k in "uvw":
        p[k] = (0.02 * rng.standard_normal(cell.size)).astype(np.float32)
    p["q"] = rng.uniform(0.5, 1.5, cell.size).astype(np.float32)
    return p


@pytest.mark.parametrize("grid", [(8, 4, 4), (16, 8, 12)])
@pytest.mark.parametrize("spread", [8, 31, 32, 33, 63, 64, 65, 66, 300])
def test_uneven_cells_vs_fp64(cuda, spread, grid):
    rng = np.random.default_rng(spread)
    wl = W.GemWorkload(name="t", nxc=grid[0], nyc=grid[1], nzc=grid[2], Lx=grid[0] * 0.5,
                       Ly=grid[1] * 0.5, Lz=grid[2] * 0.5)
    n = int(np.prod(grid))
    lone = np.zeros(n, int)
    lone[n // 2] = 1
    few = rng.integers(0, 4, n)
    few[rng.permutation(n)[:max(1, n // 40)]] += spread
    most = np.full(n, 1 + spread)
    most[::3] = 1
    parts = [at_rest(rng, wl, c.reshape(grid)) for c in (few, lone, most, few[::-1])]
    fields = [np.zeros(wl.nodes, np.float32) for _ in range(6)]
    sim = run_sim(cuda, wl, fields, parts)
    orc64 = oracle.CpuOracle("restated", 64)
    for s in range(4):
        _, m64 = oracle64(orc64, wl, fields, parts[s], wl.species[s].qom)
        err = rel_l2(sim.moments(s).cpu().numpy(), m64)
        assert (err <= 1e-5).all(), (s, err)
    sim.close()
