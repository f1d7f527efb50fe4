"""The kick and the drift as calls of their own, and the fused step, through
the pipelined kernel against the per-brick one (lf2_set_move_kernel(1)):
the same particles bit for bit, compared by id, and the same max |v|.  Row
lengths that no tensor map takes (n0 % 4 != 0) and a field off the 16-byte
boundary run from a copy of the field with aligned rows; a brick far above the
others' count is taken first; a drift needs no field and runs on any lattice."""
import numpy as np
import pytest

from tests.helpers import by_id, small_case

pytestmark = pytest.mark.gpu


def _pair(n, cell, off, vel, mass, ids):
    import latfield2_b200 as L
    out = []
    for which in (0, 1):
        ctx = L.Context(n, box=tuple(v / n[0] for v in n), mode=1)
        ctx.set_particles(cell, off, vel, mass=mass, ids=ids,
                          global_mass=0.0 if mass is not None else 1.0 / len(cell))
        ctx.set_move_kernel(which)
        out.append(ctx)
    return out


def _same(a, b, mass):
    ga, gb = (by_id(c.get_particles(mass=mass, ids=True)) for c in (a, b))
    for k in ga:
        np.testing.assert_array_equal(ga[k], gb[k])


CASES = [((32, 32, 32), 30000, False, False), ((33, 40, 37), 40000, True, True),
         ((50, 32, 48), 60000, True, False), ((16, 7, 24), 3000, False, True),
         ((35, 32, 32), 1, False, False)]


@pytest.mark.parametrize("n,npart,clustered,with_mass", CASES)
def test_separate_kick_and_drift(cuda, n, npart, clustered, with_mass):
    import torch
    cell, off, vel = small_case(n, npart, seed=11, vel_sigma=0.05, clustered=clustered)
    rng = np.random.default_rng(2)
    mass = ((1 + 0.1 * rng.random(npart)) / npart).astype(np.float32) if with_mass else None
    a, b = _pair(n, cell, off, vel, mass, np.arange(npart, dtype=np.int64))
    F = torch.from_numpy(rng.standard_normal((3, n[2], n[1], n[0])).astype(np.float32)).cuda()
    Fa, Fb = a.field(3, F), b.field(3, F)
    for _ in range(3):
        assert a.gather_kick(Fa, 0.05, want_max_v=True) == b.gather_kick(Fb, 0.05, want_max_v=True)
        a.drift_rebin(0.3)
        b.drift_rebin(0.3)
        assert a.last_max_velocity() == b.last_max_velocity()
        assert a.rebin_stats()[2] == b.rebin_stats()[2]
    _same(a, b, with_mass)
    assert a.flags() & ~0x8 == 0 and b.flags() & ~0x8 == 0


@pytest.mark.parametrize("n,npart,clustered,with_mass", CASES[1:3])
def test_step_with_other_row_lengths(cuda, n, npart, clustered, with_mass):
    import torch
    cell, off, vel = small_case(n, npart, seed=13, vel_sigma=0.05, clustered=clustered)
    rng = np.random.default_rng(3)
    mass = ((1 + 0.1 * rng.random(npart)) / npart).astype(np.float32) if with_mass else None
    a, b = _pair(n, cell, off, vel, mass, np.arange(npart, dtype=np.int64))
    F = torch.from_numpy(rng.standard_normal((3, n[2], n[1], n[0])).astype(np.float32)).cuda()
    ra, rb = a.field(1), b.field(1)
    for _ in range(3):
        a.step(a.field(3, F), 0.05, 0.3, ra)
        b.step(b.field(3, F), 0.05, 0.3, rb)
        F = F * 0.5  # another buffer and other values
    assert a.last_move_kernel() == 2 and b.last_move_kernel() == 1
    _same(a, b, with_mass)
    np.testing.assert_array_equal(ra.export_internal(), rb.export_internal())


def test_field_off_the_16_byte_boundary_and_sparse_stores(cuda):
    import torch
    n, npart = (32, 36, 40), 20000
    cell, off, vel = small_case(n, npart, seed=17, vel_sigma=0.05)
    a, b = _pair(n, cell, off, vel, None, np.arange(npart, dtype=np.int64))
    sites = 3 * n[0] * n[1] * n[2]
    buf = torch.randn(sites + 1, generator=torch.Generator().manual_seed(1)).cuda()
    F = buf[1:].view(3, n[2], n[1], n[0])
    for ctx in (a, b):
        ctx.step(ctx.field(3, F), 0.05, 0.3)
    _same(a, b, False)
    # fewer than a third of a particle per site: not worth the copy
    few = npart // 4
    c, _ = _pair((33, 36, 40), *(x[:few] for x in small_case((33, 36, 40), npart, seed=17)), None, None)
    F2 = torch.zeros(3, 40, 36, 33, device="cuda")
    c.step(c.field(3, F2), 0.05, 0.3)
    assert c.last_move_kernel() == 1


@pytest.mark.parametrize("warm", [False, True])
def test_kick_drift_and_deposit_under_capture(cuda, warm):
    """Captured calls allocate nothing (the padded rows come with the load),
    whether the context has kicked before or not.  The replayed graph moves the
    particles as the same calls outside one."""
    import torch
    import latfield2_b200 as L
    n, npart = (50, 32, 48), 60000
    cell, off, vel = small_case(n, npart, seed=19, vel_sigma=0.05, clustered=True)
    F = torch.from_numpy(np.random.default_rng(5).standard_normal((3, n[2], n[1], n[0])).astype(np.float32)).cuda()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    ctxs = []
    for stream in (None, s.cuda_stream):
        ctx = L.Context(n, box=tuple(v / n[0] for v in n), mode=1, stream=stream)
        ctx.set_particles(cell, off, vel, ids=np.arange(npart, dtype=np.int64), global_mass=1.0 / npart)
        f, rho = ctx.field(3, F), ctx.field(1)
        ctx.deposit_scalar(rho)  # (its scratch)

        def passes(ctx=ctx, f=f, rho=rho):
            ctx.gather_kick(f, 0.05)
            ctx.drift_rebin(0.3)
            ctx.deposit_scalar(rho)
        if warm:
            passes()
        ctxs.append((ctx, passes, rho))
    (a, pass_a, rho_a), (b, pass_b, rho_b) = ctxs
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        pass_b()
    for _ in range(3):
        pass_a()
        with torch.cuda.stream(s):
            graph.replay()
    torch.cuda.synchronize()
    _same(a, b, False)
    np.testing.assert_array_equal(rho_a.export_internal(), rho_b.export_internal())
    assert a.flags() & ~0x8 == 0 and b.flags() & ~0x8 == 0


def test_the_first_kick_allocates_nothing(cuda):
    """The padded rows (36 MB here) come with the load and go with the choice of
    the per-brick kernel, or with a store for which they do not pay; the first
    step takes the pipelined kernel."""
    import torch
    import latfield2_b200 as L
    n, npart = (150, 141, 142), 2300000
    cell, off, vel = small_case(n, npart, seed=23, vel_sigma=0.05)
    F = torch.zeros(3, n[2], n[1], n[0], device="cuda")
    sites = F.numel() // 3

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def fresh():
        ctx = L.Context(n, box=tuple(v / n[0] for v in n), mode=1)
        ctx.set_particles(cell, off, vel, global_mass=1.0 / npart)
        return ctx, ctx.field(3, F)
    warm, f = fresh()  # (kernels are loaded with their first launch)
    warm.gather_kick(f, 0.1)
    warm.step(f, 0.1, 0.1)
    warm.set_move_kernel(1)
    ctx, f = fresh()
    before = free()
    ctx.gather_kick(f, 0.1)
    ctx.step(f, 0.1, 0.1)
    assert ctx.last_move_kernel() == 2
    assert abs(before - free()) < 6 * sites
    ctx.set_move_kernel(1)
    assert free() - before > 6 * sites
    ctx.step(f, 0.1, 0.1)
    assert ctx.last_move_kernel() == 1
    ctx.set_move_kernel(0)
    assert abs(before - free()) < 6 * sites
    ctx.set_particles(cell[:1000], off[:1000], vel[:1000], global_mass=1.0)  # nor with a sparse store
    assert free() - before > 6 * sites
    ctx.close()
    warm.close()


@pytest.mark.parametrize("n,npart,clustered,with_mass",
                         CASES + [((64, 48, 32), 40, False, False), ((64, 48, 32), 90000, True, True)])
def test_both_kernels_of_the_separate_calls(cuda, n, npart, clustered, with_mass):
    """The kernel that the sizes do not choose here: pipelined (2) against
    per-brick (1), kick and drift each."""
    import torch
    cell, off, vel = small_case(n, npart, seed=29, vel_sigma=0.05, clustered=clustered)
    rng = np.random.default_rng(4)
    mass = ((1 + 0.1 * rng.random(npart)) / npart).astype(np.float32) if with_mass else None
    a, b = _pair(n, cell, off, vel, mass, np.arange(npart, dtype=np.int64))
    a.set_move_kernel(2)
    F = torch.from_numpy(rng.standard_normal((3, n[2], n[1], n[0])).astype(np.float32)).cuda()
    Fa, Fb = a.field(3, F), b.field(3, F)
    for _ in range(3):
        assert a.gather_kick(Fa, 0.05, want_max_v=True) == b.gather_kick(Fb, 0.05, want_max_v=True)
        a.drift_rebin(0.3)
        b.drift_rebin(0.3)
        assert a.rebin_stats()[2] == b.rebin_stats()[2]
    _same(a, b, with_mass)
    assert a.flags() & ~0x8 == 0 and b.flags() & ~0x8 == 0
