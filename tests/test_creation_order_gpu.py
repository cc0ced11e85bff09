"""Creating a simulation zeroes device memory; that zeroing has to come before what the caller
queues next, also on a stream that the default stream does not block, and also while the default
stream is busy. (Serving jobs admitted while others ran lost parts of their fields to it.)"""
import pytest

from sputnipic_b200 import workload as W

pytestmark = pytest.mark.gpu


def test_zeroing_comes_before_the_callers_stream(cuda):
    torch = cuda
    from sputnipic_b200 import device
    from sputnipic_b200.sim import Simulation

    wl = W.small_gem(nxc=16, nyc=8, nzc=8, E_amp=1e-3, species=W.gem_species((8, 8, 8, 8)))
    fields = device.gen_fields(wl)
    parts = [device.gen_particles(wl, s) for s in range(2)]
    torch.cuda.synchronize()
    st = torch.cuda.Stream()

    def moments(busy):
        if busy:
            torch.cuda._sleep(200_000_000)   # about 0.1 s of the default stream
        sim = Simulation(wl, species=[0, 1])
        sim.set_fields(fields, stream=st)
        for s, p in enumerate(parts):
            sim.load_species(s, p, stream=st)
        sim.cycle(1, stream=st)
        st.synchronize()
        torch.cuda.synchronize()   # whatever the creation left on the default stream
        sim.cycle(1, stream=st)    # and what it left of the fields
        assert sim.check(st) == 0
        out = [sim.moments(s, stream=st) for s in range(2)]
        st.synchronize()
        sim.close()
        return out

    idle = moments(False)
    for a, b in zip(idle, moments(True)):
        assert float(a.norm()) > 0
        # the same particles' FP32 cell sums in any order (the bar of the precision form)
        assert float((a - b).norm() / a.norm()) <= 1e-5


def test_moments_written_right_after_creation(cuda):
    """A new simulation's moments may be written, folded and read at once, on the default stream
    and on another one, also by a capturing stream: the zeroing comes first."""
    torch = cuda
    from sputnipic_b200.sim import Simulation

    wl = W.small_gem(nxc=128, nyc=64, nzc=64, periodic=(False, False, False))   # 47 MB a species
    ones = torch.ones(10, wl.nodes, dtype=torch.float64, device="cuda")
    want = ones.view(10, wl.nxn, wl.nyn, wl.nzn).clone()
    for axis in (1, 2, 3):
        for at in (1, want.shape[axis] - 2):
            plane = want.narrow(axis, at, 1)
            inner = [slice(None)] + [slice(1, -1) if a != axis else slice(None) for a in (1, 2, 3)]
            plane[tuple(inner)] *= 2
    torch.cuda.synchronize()
    for st in (torch.cuda.default_stream(), torch.cuda.Stream()):
        for _ in range(3):
            sim = Simulation(wl, species=[0, 1])
            with torch.cuda.stream(st):
                sim.moments_view(1).copy_(ones)
                sim.apply_bc_ids(1, stream=st)
                got = sim.moments(1, stream=st)
            st.synchronize()
            assert torch.equal(got.view_as(want), want)
            assert sim.check(st) == 0
            sim.close()
    sim = Simulation(wl, species=[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sim.apply_bc_ids(0, stream=torch.cuda.current_stream())
    sim.moments_view(0).copy_(ones)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(sim.moments_view(0).view_as(want), want)
    sim.close()


def test_reported_errors_are_cleared_for_every_stream(cuda):
    """check() clears the error word before it returns: a particle off the grid that another stream
    deposits right after it is reported, and a clean deposit then is not."""
    torch = cuda
    from sputnipic_b200 import _lib, device

    wl = W.small_gem(nxc=16, nyc=8, nzc=8, species=W.gem_species((8, 8, 8, 8)))
    bad = device.gen_particles(wl, 0)
    good = {k: v.clone() for k, v in bad.items()}
    bad["y"][7] = 1e9
    mom = torch.zeros(10, wl.nodes, device="cuda")
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    ctx = device.GridContext(wl)
    for _ in range(20):
        for st in (a, b):
            ctx.p2g(bad, mom, stream=st)
            with pytest.raises(_lib.SpbError):
                _lib.check(ctx.check(st))
    ctx.p2g(good, mom, stream=a)
    assert ctx.check(a) == 0
    ctx.close()
