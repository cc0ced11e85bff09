"""The plain deposit in cell order (65,536 particles and more) against the oracle: sizes at the
threshold and its remainders, grids smaller than a tile and longer than one, all particles in one
cell, particles on nodes and walls, a domain that does not start at 0, positions off the grid, and
more particles than one chunk holds. Bar: |gpu - ref| <= 32 eps32 sum |term| per node (the rounding
bound of a reordered float sum, as in test_parity_plain_gpu.py)."""
import numpy as np
import pytest

import oracle
from sputnipic_b200 import workload as W

pytestmark = pytest.mark.gpu
EPS32 = float(np.finfo(np.float32).eps)


def particles(rng, wl, n, where):
    p = {}
    for k, L, c in zip("xyz", (wl.Lx, wl.Ly, wl.Lz), (wl.nxc, wl.nyc, wl.nzc)):
        if where == "one cell":
            a = (c // 2 + rng.random(n)) * (L / c)
        elif where == "nodes":
            a = rng.integers(0, c + 1, n) * (L / c)
        else:
            a = rng.random(n) * L
        a = a.astype(np.float32)
        p[k] = np.where(a.astype(np.float64) > L, np.nextafter(a, np.float32(0)), a)
    for k in "uvw":
        p[k] = (0.05 * rng.standard_normal(n)).astype(np.float32)
    p["q"] = rng.uniform(-1, 1, n).astype(np.float32)
    return p


def check(got, wl, p):
    setup = oracle.setup_from(wl)
    ref = [np.zeros(wl.nodes, np.float32) for _ in range(10)]
    oracle.CpuOracle("restated", 32).interp_p2g(setup, p, ref)
    a = {k: (np.abs(p[k]) if k in "uvwq" else p[k]).astype(np.float64) for k in "xyzuvwq"}
    absm = [np.zeros(wl.nodes) for _ in range(10)]
    oracle.CpuOracle("restated", 64).interp_p2g(setup, a, absm)
    bad = np.abs(got.astype(np.float64) - np.stack(ref)) > 32 * EPS32 * np.stack(absm) + 1e-30
    assert not bad.any(), f"{bad.sum()} moment entries outside the bound"


def on_gpu(torch, p):
    return {k: torch.from_numpy(v.copy()).cuda() for k, v in p.items()}


@pytest.mark.parametrize("n", [65535, 65536, 70001])
@pytest.mark.parametrize("grid", [(1, 1, 1), (1, 1, 300), (17, 5, 9), (40, 24, 16)])
@pytest.mark.parametrize("where", ["anywhere", "one cell", "nodes"])
def test_against_oracle(cuda, n, grid, where):
    torch = cuda
    from sputnipic_b200 import device
    rng = np.random.default_rng(n + grid[2])
    wl = W.GemWorkload(name="t", nxc=grid[0], nyc=grid[1], nzc=grid[2], Lx=grid[0] * 0.3,
                       Ly=grid[1] * 0.25, Lz=grid[2] * 0.7)
    p = particles(rng, wl, n, where)
    ctx = device.GridContext(wl)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    ctx.p2g(on_gpu(torch, p), mom)
    assert ctx.check() == 0
    check(mom.cpu().numpy(), wl, p)
    once = mom.clone()
    ctx.p2g(on_gpu(torch, p), mom)   # a second call adds
    assert torch.allclose(mom, 2 * once, rtol=1e-4, atol=1e-5 * float(once.abs().max()))
    ctx.close()


def test_shifted_domain_and_off_grid(cuda):
    torch = cuda
    from sputnipic_b200 import device, dropin
    rng = np.random.default_rng(3)
    wl = W.GemWorkload(name="t", nxc=12, nyc=10, nzc=7, Lx=3.0, Ly=2.5, Lz=1.75)   # cells of 0.25
    n = 66000
    p = particles(rng, wl, n, "anywhere")
    for k in "xyz":   # multiples of 2^-18: shifting by 0.5 is exact
        p[k] = (np.floor(p[k] * 2 ** 18) / 2 ** 18).astype(np.float32)
    grd = dropin.setGrid(dropin.make_parameters(wl))
    grd.xStart = grd.yStart = grd.zStart = 0.5
    for a in ("XN", "YN", "ZN"):
        grd._arrays[a] += np.float32(0.5)
    ctx = device.GridContext(grid=grd)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    moved = {k: (v + np.float32(0.5) if k in "xyz" else v) for k, v in p.items()}
    ctx.p2g(on_gpu(torch, moved), mom)
    assert ctx.check() == 0
    check(mom.cpu().numpy(), wl, p)
    ctx.close()
    # positions off the node array are flagged and clamped, on both paths
    from sputnipic_b200 import _lib
    for shift in (0.0, 0.5):
        ctx = device.GridContext(wl) if shift == 0.0 else device.GridContext(grid=grd)
        for bad in (1e9, -1e9, float("nan")):
            q = on_gpu(torch, p)
            q["y"][5] = bad
            ctx.p2g(q, mom)
            with pytest.raises(_lib.SpbError):
                _lib.check(ctx.check())
        ctx.close()


def test_more_than_one_chunk(cuda):
    torch = cuda
    from sputnipic_b200 import device
    wl = W.GemWorkload(name="t", nxc=32, nyc=32, nzc=32, Lx=8.0, Ly=8.0, Lz=8.0)
    n = (1 << 26) + 100_001
    g = torch.Generator(device="cuda").manual_seed(1)
    p = {k: torch.rand(n, generator=g, device="cuda") * (8.0 if k in "xyz" else 0.1) for k in "xyzuvwq"}
    ctx = device.GridContext(wl)
    whole = torch.zeros(10, wl.nodes, device="cuda")
    ctx.p2g(p, whole)
    parts = torch.zeros(10, wl.nodes, device="cuda")
    for a, b in ((0, n // 3), (n // 3, n)):
        ctx.p2g({k: v[a:b].contiguous() for k, v in p.items()}, parts)
    assert ctx.check() == 0
    # all terms positive: two FP32 sums of the same 2048 * 8 terms a node
    assert float(((whole - parts).norm(dim=1) / whole.norm(dim=1)).max()) < 2e-6
    ctx.close()


@pytest.mark.parametrize("u", [3e19, float("inf"), float("-inf"), float("nan")])
def test_infinite_products_stay_infinite(cuda, u):
    """A velocity whose square overflows (or that is not finite) gives infinity and NaN in the
    moments and at the nodes where the reference has them, whatever the counts of the other cells."""
    torch = cuda
    from sputnipic_b200 import device
    rng = np.random.default_rng(5)
    wl = W.GemWorkload(name="t", nxc=16, nyc=8, nzc=8, Lx=4.0, Ly=2.0, Lz=2.0)
    p = particles(rng, wl, 66000, "anywhere")
    # a cell of 24 such particles beside cells of about 64 others (in up to 8 parts)
    p["x"][(p["x"] > 1.0) & (p["x"] < 1.25)] += np.float32(1.0)
    for k, at in (("x", 1.1), ("y", 0.6), ("z", 0.9), ("u", u), ("v", 0.05), ("w", 0.1), ("q", 0.5)):
        p[k][:24] = at
    p["x"][:24] += np.arange(24, dtype=np.float32) / 256
    ref = np.zeros((10, wl.nodes), np.float32)
    oracle.CpuOracle("restated", 32).interp_p2g(oracle.setup_from(wl), p, list(ref))
    ctx = device.GridContext(wl)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    ctx.p2g(on_gpu(torch, p), mom)
    assert ctx.check() == 0
    got = mom.cpu().numpy()
    ctx.close()
    assert not np.isfinite(ref).all()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(np.where(np.isinf(got), got, 0), np.where(np.isinf(ref), ref, 0))


def test_equal_charges_in_one_cell(cuda):
    """Four million equal particles in one cell: every rounding of a running FP32 sum then falls the
    same way. Bar: runs of 16 (8 eps32), a tree of 5, at most 2,048 partial sums one after another
    (1,024) and the terms' own roundings (8); one sum per lane of a warp is off by 3,300."""
    torch = cuda
    from sputnipic_b200 import device
    wl = W.GemWorkload(name="t", nxc=16, nyc=16, nzc=16, Lx=4.0, Ly=4.0, Lz=4.0)
    n, q, u = 1 << 22, float(np.float32(0.77)), (0.3, -0.2, 0.1)
    p = {k: torch.full((n,), 2.125, device="cuda") for k in "xyz"}   # the cell's centre
    p.update({k: torch.full((n,), a, device="cuda") for k, a in zip("uvw", u)}, q=None)
    p["q"] = torch.full((n,), q, device="cuda")
    ctx = device.GridContext(wl)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    ctx.p2g(p, mom)
    assert ctx.check() == 0
    ctx.close()
    a, b, c = (float(np.float32(v)) for v in u)
    want = n * q * 8 * np.array([1, a, b, c, a * a, a * b, a * c, b * b, b * c, c * c])
    got = mom.double().cpu().numpy().reshape(10, wl.nxn, wl.nyn, wl.nzn)
    cell = got[:, 9:11, 9:11, 9:11].reshape(10, 8)
    assert (np.abs(cell / want[:, None] - 1) <= 1042.5 * EPS32).all()
    assert np.count_nonzero(got) == 80


def check64(got, wl, p, bar):
    """|gpu - FP64| <= bar eps32 sum |term| per node."""
    setup = oracle.setup_from(wl)
    o64 = oracle.CpuOracle("restated", 64)
    ref, absm = ([np.zeros(wl.nodes) for _ in range(10)] for _ in range(2))
    d = {k: p[k].astype(np.float64) for k in "xyzuvwq"}
    o64.interp_p2g(setup, d, ref)
    o64.interp_p2g(setup, {k: (np.abs(v) if k in "uvwq" else v) for k, v in d.items()}, absm)
    err = np.abs(got.astype(np.float64) - np.stack(ref))
    worst = (err / (EPS32 * np.stack(absm) + 1e-30)).max()
    assert worst <= bar, worst


@pytest.mark.parametrize("grid", [(1, 1, 1), (4, 4, 4), (1, 1, 300), (40, 24, 16)])
@pytest.mark.parametrize("where", ["anywhere", "a third in one cell", "one cell", "sizes"])
def test_clumps_and_tiny_grids(cuda, grid, where):
    """Millions of particles on few cells, or in one cell of many, and cells at the counts where the
    split of their records changes. Cells are 1/4 wide, so node distances are exact; a term has at
    most 8 roundings, a sum runs of 16 and a tree of 5 (random ones: under 8 eps32), and a node at
    most 2,400 FP32 adds of partial sums, random in sign: 0.29 sqrt(2400 / 3) < 9 eps32."""
    torch = cuda
    from sputnipic_b200 import device
    rng = np.random.default_rng(sum(grid))
    wl = W.GemWorkload(name="t", nxc=grid[0], nyc=grid[1], nzc=grid[2], Lx=grid[0] * 0.25,
                       Ly=grid[1] * 0.25, Lz=grid[2] * 0.25)
    n = (1 << 21) + 5
    p = particles(rng, wl, n, "anywhere")
    held = {"a third in one cell": [n // 3], "one cell": [n],
            "sizes": [1023, 1024, 1025, 2047, 2048, 2049, 4097, 100_000, 300_001]}.get(where, [])
    at = 0
    for m in held:
        for k, c in zip("xyz", grid):
            p[k][at:at + m] = (rng.integers(0, c) + rng.random(m)).astype(np.float32) * 0.25
        at += m
    for k, L in zip("xyz", (wl.Lx, wl.Ly, wl.Lz)):
        p[k] = np.minimum(p[k], np.nextafter(np.float32(L), np.float32(0)))
    order = rng.permutation(n)
    p = {k: v[order] for k, v in p.items()}
    ctx = device.GridContext(wl)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    ctx.p2g(on_gpu(torch, p), mom)
    assert ctx.check() == 0
    check64(mom.cpu().numpy(), wl, p, 32)
    ctx.close()


@pytest.mark.parametrize("busy", [1, 31, 32, 33, 128])
@pytest.mark.parametrize("most", [1, 16, 17])
def test_sparse_tiles(cuda, busy, most):
    """Tiles with few cells that hold particles, and few particles in each, on both sides of the
    counts from which their cells' sums go through the node sums."""
    torch = cuda
    from sputnipic_b200 import device
    rng = np.random.default_rng(busy)
    wl = W.GemWorkload(name="t", nxc=80, nyc=40, nzc=40, Lx=20.0, Ly=10.0, Lz=10.0)
    cells = np.indices((80, 40, 40)).reshape(3, -1).T.reshape(10, 8, 10, 4, 10, 4, 3)
    tiles = cells.transpose(0, 2, 4, 1, 3, 5, 6).reshape(1000, 128, 3)
    at = np.concatenate([t[rng.permutation(128)[:busy]] for t in tiles])
    count = rng.integers(1, most + 1, len(at))
    count[0] = most
    at = np.repeat(at, count, axis=0)
    lone = 65_536 - len(at)   # a first inner tile with everything that is missing
    if lone > 0:
        at = np.concatenate([at, tiles[0][rng.integers(0, 128, lone)]])
    p = {k: ((at[:, a] + rng.uniform(0, 0.999, len(at))) * 0.25).astype(np.float32)
         for a, k in enumerate("xyz")}
    for k in "uvw":
        p[k] = (0.05 * rng.standard_normal(len(at))).astype(np.float32)
    p["q"] = rng.uniform(-1, 1, len(at)).astype(np.float32)
    ctx = device.GridContext(wl)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    ctx.p2g(on_gpu(torch, p), mom)
    assert ctx.check() == 0
    check(mom.cpu().numpy(), wl, p)
    ctx.close()


@pytest.mark.parametrize("grid", [(1, 40, 33), (2, 31, 64), (40, 1, 33), (33, 2, 40), (40, 33, 1),
                                  (31, 64, 2), (3, 20, 20), (4, 40, 40)])
@pytest.mark.parametrize("where", ["anywhere", "one cell", "nodes"])
def test_thin_grids(cuda, grid, where):
    """Grids a few cells thin along each axis: the tiles of one layer, and those next to the rule."""
    torch = cuda
    from sputnipic_b200 import device
    wl = W.GemWorkload(name="t", nxc=grid[0], nyc=grid[1], nzc=grid[2], Lx=grid[0] * 0.25,
                       Ly=grid[1] * 0.25, Lz=grid[2] * 0.25)
    p = particles(np.random.default_rng(sum(grid)), wl, 70_001, where)
    ctx = device.GridContext(wl)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    ctx.p2g(on_gpu(torch, p), mom)
    assert ctx.check() == 0
    check(mom.cpu().numpy(), wl, p)
    ctx.close()


@pytest.fixture
def small_pool(cuda):
    """The device's memory pool replaced by one of 32 MB, of which `held` bytes are taken."""
    from contextlib import contextmanager

    from cuda.bindings import runtime as rt

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) > 1 else None

    @contextmanager
    def replaced(held):
        props = rt.cudaMemPoolProps()
        props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
        props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
        props.location.id = 0
        props.maxSize = 32 << 20
        cuda.cuda.synchronize()
        pool = ok(rt.cudaMemPoolCreate(props))
        taken = ok(rt.cudaMallocFromPoolAsync(held, pool, 0)) if held else None
        ok(rt.cudaDeviceSetMemPool(0, pool))
        try:
            yield
        finally:
            cuda.cuda.synchronize()
            ok(rt.cudaDeviceSetMemPool(0, ok(rt.cudaDeviceGetDefaultMemPool(0))))
            if taken is not None:
                ok(rt.cudaFreeAsync(taken, 0))
            cuda.cuda.synchronize()
            ok(rt.cudaMemPoolDestroy(pool))
    return replaced


@pytest.fixture(params=["accumulator", "direct"])
def deposit_mode(request):
    from sputnipic_b200.device import set_plain_deposit_mode
    prev = set_plain_deposit_mode(request.param)
    yield request.param
    set_plain_deposit_mode(prev)


def launches():
    from sputnipic_b200 import _lib
    return _lib.load().spb_launch_count()


@pytest.mark.parametrize("where", ["anywhere", "one cell"])
def test_without_scratch(cuda, small_pool, deposit_mode, where):
    """Scratch for half the particles: two chunks. None: the deposit of smaller batches, into the
    accumulator (and its fold) or straight into the moments, as the mode says."""
    torch = cuda
    from sputnipic_b200 import device
    wl = W.GemWorkload(name="t", nxc=16, nyc=8, nzc=8, Lx=4.0, Ly=2.0, Lz=2.0)
    ctx = device.GridContext(wl)
    for n, held, want in ((1_500_000, 0, 8),
                          (70_001, 31 << 20, 2 if deposit_mode == "accumulator" else 1)):
        p = particles(np.random.default_rng(n), wl, n, where)
        d, mom = on_gpu(torch, p), torch.zeros(10, wl.nodes, device="cuda")
        with small_pool(held):
            before = launches()
            ctx.p2g(d, mom)
            assert launches() - before == want
        assert ctx.check() == 0
        if n < 100_000:
            check(mom.cpu().numpy(), wl, p)
        else:
            whole = torch.zeros_like(mom)
            ctx.p2g(d, whole)
            # the same terms in runs of 16 and partial sums of other parts
            assert float(((mom - whole).norm(dim=1) / whole.norm(dim=1)).max()) < 2e-6
    ctx.close()


def test_pipeline_without_scratch(cuda, small_pool, deposit_mode):
    """interpP2G of host arrays of more than one pipeline chunk (2^22 particles), none of which gets
    scratch: an accumulator per stream, each folded once."""
    from sputnipic_b200 import dropin
    dropin.release_all()
    dropin.set_residency(False)
    wl = W.GemWorkload(name="t", nxc=16, nyc=8, nzc=8, Lx=4.0, Ly=2.0, Lz=2.0)
    n = (1 << 22) + 100_000
    p = particles(np.random.default_rng(2), wl, n, "anywhere")
    p["q"] = np.abs(p["q"])
    p["u"], p["v"], p["w"] = (np.abs(p[k]) for k in "uvw")
    setup = oracle.setup_from(wl)
    ref32 = [np.zeros(wl.nodes, np.float32) for _ in range(10)]
    oracle.CpuOracle("restated", 32).interp_p2g(setup, p, ref32)
    ref = [np.zeros(wl.nodes) for _ in range(10)]
    oracle.CpuOracle("restated", 64).interp_p2g(
        setup, {k: p[k].astype(np.float64) for k in "xyzuvwq"}, ref)
    param = dropin.make_parameters(wl)
    grd = dropin.setGrid(param)
    part = dropin.particle_allocate(param, 0, arrays=p)
    ids = dropin.interp_dens_species_allocate(grd, 0)
    with small_pool(31 << 20):
        before = launches()
        dropin.interpP2G(part, ids, grd, raise_on_error=True)
        assert launches() - before == (4 if deposit_mode == "accumulator" else 2)
    # 33,000 positive terms a node, most added one by one as the reference's FP32 code does
    for got, r32, r in zip(dropin.moments(ids), ref32, ref):
        err = np.linalg.norm(got.ravel() - r), np.linalg.norm(r32 - r)
        assert err[0] <= 2 * err[1] + 1e-7 * np.linalg.norm(r)
    dropin.release_all()


@pytest.mark.parametrize("grid,n", [((40, 24, 16), 1000), ((40, 24, 16), 65535),
                                    ((40, 24, 16), 65536), ((64, 64, 64), 70_000),
                                    ((64, 64, 64), 150_381), ((64, 64, 64), 150_382)])
@pytest.mark.parametrize("where", ["anywhere", "one cell"])
def test_mover_interp_in_one_pass_and_in_two(cuda, grid, n, where):
    """mover_interp on both sides of its rule (65,536 particles, half a particle per node): the
    particles that mover gives, bit for bit, and their moments."""
    torch = cuda
    from sputnipic_b200 import device
    wl = W.GemWorkload(name="t", nxc=grid[0], nyc=grid[1], nzc=grid[2], Lx=grid[0] * 0.25,
                       Ly=grid[1] * 0.25, Lz=grid[2] * 0.25, E_amp=1e-3)
    p = particles(np.random.default_rng(n), wl, n, where)
    one_pass = n < 65536 or 2 * n < wl.nodes
    ctx = device.GridContext(wl)
    ctx.set_fields(device.gen_fields(wl))
    push = device.push_params(wl, 1)
    moved, both = on_gpu(torch, p), on_gpu(torch, p)
    ctx.mover(moved, push)
    mom = torch.zeros(10, wl.nodes, device="cuda")
    before = launches()
    ctx.mover_interp(both, push, mom)
    assert launches() - before == (2 if one_pass else 5)
    assert ctx.check() == 0
    for k in "xyzuvw":
        assert torch.equal(moved[k], both[k])
    check(mom.cpu().numpy(), wl, {k: v.cpu().numpy() for k, v in both.items()})
    ctx.close()
