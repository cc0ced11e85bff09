"""The mover forms its cell indices, its reciprocal, its final velocities and its boundary tests in
float where that gives the reference's bits. Checked bit for bit against the oracle where it could
fail: positions a few ulps around nodes and walls, spacings that are no floats, momenta from far
below to far above 1 in omdtsq, and (general path) a domain that does not start at 0."""
import numpy as np
import pytest

import oracle
from sputnipic_b200 import dropin
from sputnipic_b200 import workload as W

pytestmark = pytest.mark.gpu


def around(rng, n, cells, d, L):
    """Positions on nodes and walls, up to three floats to either side, inside [0, L]."""
    p = (rng.integers(0, cells + 1, n) * d).astype(np.float32)
    for _ in range(3):
        k = rng.integers(-1, 2, n)
        p = np.where(k < 0, np.nextafter(p, np.float32(-1)), np.where(
            k > 0, np.nextafter(p, np.float32(2 * L)), p))
    free = rng.random(n) < 0.3
    p = np.where(free, (rng.random(n) * L).astype(np.float32), p)
    top = np.float32(L)
    top = np.nextafter(top, np.float32(0)) if float(top) > L else top
    return np.clip(p, np.float32(0), top).astype(np.float32)


@pytest.mark.parametrize("variant", ["mover", "moverv"])
@pytest.mark.parametrize("grid,L,niter,per", [
    ((61, 7, 33), (20.0, 3.1, 7.7), 3, (True, False, True)),
    ((5, 48, 3), (0.9, 15.0, 1.0), 1, (False, False, False)),
    ((16, 9, 11), (10.0, 1e-3, 1e3), 4, (True, True, True)),
])
def test_mover_float_paths_bit_identical(cuda, grid, L, niter, per, variant):
    rng = np.random.default_rng(niter)
    wl = W.GemWorkload(name="t", nxc=grid[0], nyc=grid[1], nzc=grid[2], Lx=L[0], Ly=L[1], Lz=L[2],
                       niter=niter, periodic=per)
    n = 40000
    d = [l / c for l, c in zip(L, grid)]
    # B from 1e-8 to 10 times what turns omdtsq to 1; E moves a particle by at most 0.3 cells of
    # the finest axis
    qom = -64.0
    h = abs(qom) * 0.5 * wl.dt
    mag = 10.0 ** rng.uniform(-8, 1, wl.nodes) / h
    fields = [(min(d) * 0.3 / h / wl.dt * rng.uniform(-1, 1, wl.nodes)).astype(np.float32)
              for _ in range(3)]
    fields += [(mag * rng.uniform(-1, 1, wl.nodes)).astype(np.float32) for _ in range(3)]
    part = {k: around(rng, n, c, dd, l) for k, c, dd, l in zip("xyz", grid, d, L)}
    for k in "uvw":   # at most 0.4 cells of the finest axis a step, however B turns them
        part[k] = (0.4 * min(d) / 3 ** 0.5 / wl.dt * rng.uniform(-1, 1, n)).astype(np.float32)
        part[k][: n // 20] = 0.0
    part["q"] = np.ones(n, np.float32)
    ref = {k: v.copy() for k, v in part.items()}
    orc = oracle.CpuOracle("restated", 32)
    getattr(orc, "mover_pc" if variant == "mover" else "mover_pc_v")(
        oracle.setup_from(wl), fields, ref, qom)
    param = dropin.make_parameters(wl, ns=1)
    grd = dropin.setGrid(param)
    P = dropin.particle_allocate(param, 0, arrays=part)
    P.qom = qom
    fn = dropin.mover_PC if variant == "mover" else dropin.mover_PC_V
    assert fn(P, dropin.field_allocate(grd, fields), grd, param, raise_on_error=True) == 0
    out = dropin.particle_arrays(P)
    for k in "xyzuvw":
        bad = out[k].view(np.int32) != ref[k].view(np.int32)
        assert not bad.any(), f"{k}: {bad.sum()} of {n} differ"
    dropin.release_all()


def test_general_cells_agree_with_float_cells(cuda):
    """A domain shifted by 0.5 (node coordinates and positions shifted alike, exactly): the general
    path's double cell index on one side, the float one on the other."""
    rng = np.random.default_rng(5)
    wl = W.GemWorkload(name="t", nxc=16, nyc=8, nzc=8, Lx=4.0, Ly=2.0, Lz=2.0,
                       periodic=(True, True, True))
    fields = [(1e-3 * rng.uniform(-1, 1, wl.nodes)).astype(np.float32) for _ in range(6)]
    n = 20000
    # multiples of 2^-18 well inside the domain, so that the shift is exact
    part = {k: (rng.integers(2 ** 17, int(l * 2 ** 18) - 2 ** 17, n) / 2 ** 18).astype(np.float32)
            for k, l in zip("xyz", (4.0, 2.0, 2.0))}
    for k in "uvw":
        part[k] = np.zeros(n, np.float32)
    part["q"] = np.ones(n, np.float32)
    vel = []
    for shift in (0.0, 0.5):
        param = dropin.make_parameters(wl, ns=1)
        param.n_sub_cycles = 1
        grd = dropin.setGrid(param)
        p = {k: v.copy() for k, v in part.items()}
        if shift:
            grd.xStart = grd.yStart = grd.zStart = shift
            grd.Lx, grd.Ly, grd.Lz = 4.5, 2.5, 2.5
            for a in ("XN", "YN", "ZN"):
                grd._arrays[a] += np.float32(shift)
            for k in "xyz":
                p[k] += np.float32(shift)
        P = dropin.particle_allocate(param, 0, arrays=p)
        P.qom, P.NiterMover = 1.0, 1   # one gather, at the exactly shifted position
        dropin.mover_PC(P, dropin.field_allocate(grd, fields), grd, param, raise_on_error=True)
        vel.append({k: dropin.particle_arrays(P)[k].copy() for k in "uvw"})
        dropin.release_all()
    for k in "uvw":
        assert np.array_equal(vel[0][k], vel[1][k])
