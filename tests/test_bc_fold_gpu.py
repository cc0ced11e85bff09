"""applyBCids in one launch: bit-identical to the oracle's step-by-step fold, FP32 and FP64, for
every mix of periodic and other axes, down to one cell per axis (both boundary planes adjacent)."""
import itertools

import numpy as np
import pytest

import oracle
from sputnipic_b200 import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 1, 3), (1, 6, 2), (5, 4, 7), (34, 18, 10)])
def test_bc_fold_bit_identical(cuda, grid):
    torch = cuda
    from sputnipic_b200 import device
    from sputnipic_b200.sim import Simulation
    rng = np.random.default_rng(3)
    for per in itertools.product((False, True), repeat=3):
        wl = W.small_gem(nxc=grid[0], nyc=grid[1], nzc=grid[2], periodic=per)
        setup = oracle.setup_from(wl)
        m32 = rng.standard_normal((10, wl.nodes)).astype(np.float32)
        ref = m32.copy()
        oracle.CpuOracle("restated", 32).apply_bc_ids(setup, list(ref))
        ctx = device.GridContext(wl)
        got = torch.from_numpy(m32).cuda()
        ctx.apply_bc_ids(got, per)
        assert np.array_equal(got.cpu().numpy(), ref), (grid, per)
        ctx.close()
        if any(n % 2 for n in grid):
            continue
        m64 = rng.standard_normal((10, wl.nodes))
        ref = m64.copy()
        oracle.CpuOracle("restated", 64).apply_bc_ids(setup, list(ref))
        sim = Simulation(wl, tile=(2, 2, 2), species=[0])
        view = sim.moments_view(0)
        view.copy_(torch.from_numpy(m64))
        sim.apply_bc_ids(0)
        assert np.array_equal(view.cpu().numpy(), ref), (grid, per)
        sim.close()
