"""The differentiable chain's kernels on clustered particles: warps whose
lanes share a cell, bricks that several CTAs deposit, and the step into new
arrays and its adjoint as one call."""
import pytest

from oracle import pm_chain as P
from tests.test_gpu_adjoint import _rel

pytestmark = pytest.mark.gpu


def _sorted_case(n, mode, seed=4):
    """Particles sorted by brick and cell: a uniform background, a cell of 3000,
    a brick of 20,000 and runs of 1 to 40 particles of one cell."""
    import torch
    import latfield2_b200 as L
    from latfield2_b200.autodiff import _Ops
    g = torch.Generator(device="cpu").manual_seed(seed)

    def rand(k):
        return torch.rand(k, 3, generator=g, dtype=torch.float64)
    pos = [rand(4000) * n, rand(3000) + torch.tensor([5.0, n - 1.0, 3.0]), rand(20000) * 16 + 16]
    for k in range(1, 41):
        pos.append(rand(k) + torch.tensor([float(k % n), float((7 * k) % n), 0.0]))
    pos = (torch.cat(pos) / n % 1.0).cuda()
    npart = pos.shape[0]
    vel = (0.02 * torch.randn(npart, 3, generator=g, dtype=torch.float64)).cuda()
    m = ((1 + 0.5 * torch.rand(npart, generator=g, dtype=torch.float64)) / npart).cuda()
    ctx = L.Context((n, n, n), box=1.0, mode=L.DEPOSIT_FIXED64 if mode == "fixed" else L.DEPOSIT_FP32)
    ops = _Ops(ctx)
    key, rec = ops.state_pack(pos, vel, m, float(n))
    cell, off, v32, m32 = ops.state_unpack(torch.argsort(key), rec)
    ops.bricks = ops.brick_start(cell)
    c = cell.long()
    posd = (torch.stack([c % n, (c // n) % n, c // (n * n)], 1).double() + off.double()) / n
    return ctx, ops, cell, off, v32, m32, posd


@pytest.mark.parametrize("n", [32, 40])
@pytest.mark.parametrize("mode", ["fixed", "fp32"])
@pytest.mark.parametrize("masses", [True, False])
def test_tiled_deposit_of_dense_cells_and_bricks(cuda, n, mode, masses):
    """1e-6 of FP64 per vertex: integer sums in both modes, the terms' three
    FP32 roundings (fp32) or 2^-24 relative masses (fixed) and one of the sum."""
    import torch
    ctx, ops, cell, off, v32, m32, posd = _sorted_case(n, mode)
    npart = cell.numel()
    rho = torch.zeros(n ** 3, device="cuda")
    if masses:
        ops.deposit(cell, off, m32, rho)
        mass = m32.double()
    else:
        from latfield2_b200.autodiff import _check, _p
        _check(ctx, ops.lib.lf2_pm_deposit_bricks(ctx.h, npart, _p(cell), _p(off), None, 1.0 / npart,
                                                  _p(ops.bricks), _p(rho)), "deposit")
        mass = torch.full((npart,), 1.0 / npart, dtype=torch.float64, device="cuda")
    ref = P.deposit(posd, mass, (n, n, n))
    sel = ref > 1e-2 * ref.mean()
    assert float(((rho.double() - ref).abs() / ref)[sel].max()) <= 1e-6
    assert float((rho.double() - ref).abs().max()) <= 1e-6 * float(ref.max())


@pytest.mark.parametrize("n", [32, 40])
def test_step_adjoint_equals_its_parts(cuda, n):
    """lf2_pm_step_adjoint against the drift's and the kick's adjoint in torch
    and lf2_pm_gather_adjoint, and both against FP64 autograd of the gather
    (2e-5 of the norm, as the single adjoint kernels)."""
    import torch
    ctx, ops, cell, off, v32, m32, posd = _sorted_case(n, "fp32")
    npart, dt = cell.numel(), 0.07
    g = torch.Generator(device="cpu").manual_seed(5)
    F4 = torch.randn(4 * n ** 3, generator=g).cuda()
    g_off0, g_v0 = torch.randn(npart, 3, generator=g).cuda(), torch.randn(npart, 3, generator=g).cuda()
    a_off, a_v, a_F = g_off0.clone(), g_v0.clone(), torch.zeros(4 * n ** 3, device="cuda")
    ops.step_adj(cell, off, F4, dt, a_v, a_off, a_F)
    b_off, b_F = g_off0.clone(), torch.zeros(4 * n ** 3, device="cuda")
    b_v = g_v0 + (dt / ctx.res) * g_off0
    gG = (dt * b_v).contiguous()
    ops.gather_adj(cell, off, F4, gG, b_F, b_off)
    assert torch.equal(a_v, b_v) and torch.equal(a_off, b_off)
    assert _rel(a_F, b_F) < 1e-6  # FP32 atomics in two orders
    x = posd.clone().requires_grad_(True)
    F = F4.view(-1, 4)[:, :3].double().t().contiguous().requires_grad_(True)
    (P.gather(x, F, (n, n, n)) * gG.double()).sum().backward()
    assert _rel(a_F.view(-1, 4)[:, :3].t(), F.grad) < 2e-5
    assert _rel(a_off - g_off0, x.grad / n) < 2e-5


def test_step_into_new_arrays(cuda):
    import torch
    n = 32
    ctx, ops, cell, off, v32, m32, _ = _sorted_case(n, "fp32")
    F4 = torch.randn(4 * n ** 3, generator=torch.Generator(device="cpu").manual_seed(3)).cuda()
    v32 *= 20
    old = (cell.clone(), off.clone(), v32.clone())
    new = ops.next_state(cell, off, v32, F4, 0.05)
    for x, y in zip((cell, off, v32), old):
        assert torch.equal(x, y)
    ops.step(cell, off, v32, F4, 0.05)
    for x, y in zip((cell, off, v32), new):
        assert torch.equal(x, y)
    assert int((cell != old[0]).sum()) > 1000


def test_loss_and_its_adjoint(cuda):
    """The FP64 loss, and its adjoint against the deposit's adjoint for the
    scaled weights (the same bits, written instead of added); weights of
    another size or device are refused as torch.dot refuses them."""
    import torch
    n = 40
    ctx, ops, cell, off, v32, m32, _ = _sorted_case(n, "fp32")
    g = torch.Generator(device="cpu").manual_seed(6)
    w, rho = torch.randn(n ** 3, generator=g).cuda(), torch.randn(n ** 3, generator=g).cuda()
    want = float(torch.dot(w.double(), rho.double()))
    assert float(ops.loss(w, rho)) == pytest.approx(want, rel=1e-12, abs=1e-12 * n ** 3)
    g_off, g_v, g_m = ops.loss_adj(cell, off, m32, w, -1.7)
    want_off, want_m = torch.zeros_like(g_off), torch.zeros_like(g_m)
    ops.deposit_adj(cell, off, m32, (w * -1.7).contiguous(), want_off, want_m)
    assert torch.equal(g_off, want_off) and torch.equal(g_m, want_m) and not g_v.any()
    for bad in (w[:-1].contiguous(), w.cpu()):
        with pytest.raises(RuntimeError):
            ops.loss(bad, rho)


def test_records_off_the_32_byte_boundary(cuda):
    """32-byte records at an address that is a multiple of 16 only: the packed
    state and the unordered gradients are the same bits as at one of 32."""
    import torch
    from latfield2_b200.autodiff import _check, _p
    n, npart = 32, 5001
    ctx, ops = _sorted_case(n, "fp32")[:2]
    g = torch.Generator(device="cpu").manual_seed(8)
    pos, vel = (torch.rand(npart, 3, generator=g, dtype=torch.float64).cuda() for _ in range(2))
    m = torch.rand(npart, generator=g, dtype=torch.float64).cuda()
    key, rec = ops.state_pack(pos, vel, m, float(n))
    order = torch.argsort(key)
    want = ops.state_unpack(order, rec)
    room = torch.empty(npart * 8 + 8, dtype=torch.int32, device="cuda")
    off16 = room[4 if room.data_ptr() % 32 == 0 else 0:][:npart * 8]
    assert off16.data_ptr() % 32 == 16
    key2 = torch.empty_like(key)
    _check(ctx, ops.lib.lf2_pm_state_pack(ctx.h, npart, _p(pos), _p(vel), _p(m), float(n), _p(key2),
                                          _p(off16)), "pack")
    assert torch.equal(key, key2) and torch.equal(rec, off16)
    for x, y in zip(ops.state_unpack(order, off16), want):
        assert torch.equal(x, y)
    g_off, g_v = torch.randn(npart, 3, generator=g).cuda(), torch.randn(npart, 3, generator=g).cuda()
    g_m = torch.randn(npart, generator=g).cuda()
    ref = ops.grads_unorder(order, g_off, g_v, g_m, float(n))
    out = [torch.empty_like(x) for x in ref]
    _check(ctx, ops.lib.lf2_pm_grads_unorder(ctx.h, npart, _p(order), _p(g_off), _p(g_v), _p(g_m),
                                             float(n), _p(off16), *[_p(x) for x in out]), "grads")
    for x, y in zip(out, ref):
        assert torch.equal(x, y)


def test_chain_keeps_no_state_beside_its_checkpoints(cuda):
    """Forward and backward with a checkpoint every 4 steps: between two of them
    only the running state lives (28 bytes per particle), as its loss, the same
    in fixed point whatever the interval, is reached in place."""
    import torch
    import latfield2_b200 as L
    from latfield2_b200.autodiff import pm_chain_loss
    n, npart = 32, 400000
    g = torch.Generator(device="cpu").manual_seed(7)
    ctx = L.Context((n, n, n), box=1.0, mode=L.DEPOSIT_FIXED64)
    pos = torch.rand(npart, 3, generator=g, dtype=torch.float64).cuda()
    vel = (0.02 * torch.randn(npart, 3, generator=g, dtype=torch.float64)).cuda()
    m = torch.full((npart,), 1.0 / npart, dtype=torch.float64, device="cuda")
    S = (0.02 * torch.randn(81, generator=g, dtype=torch.float64)).cuda()
    w = torch.randn(n ** 3, generator=g, dtype=torch.float64).cuda()

    def run(every):
        leaves = [t.clone().requires_grad_(True) for t in (pos, vel, m, S, w)]
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        base = torch.cuda.memory_allocated()
        loss = pm_chain_loss(ctx, *leaves, steps=8, dt=0.02, checkpoint_every=every)
        peak = torch.cuda.max_memory_allocated() - base
        return loss, torch.autograd.grad(loss, leaves), peak
    run(4)
    loss, grads, peak = run(4)
    fields = 8 * 5 * 4 * n ** 3 + 3 * 4 * n ** 3
    # order and masses, two checkpoints and the running state, with half a state to spare
    assert peak <= (8 + 4 + 3.5 * 28) * npart + fields, peak / npart
    loss1, grads1, _ = run(1)
    assert torch.equal(loss.detach(), loss1.detach())
    for a, b in zip(grads, grads1):
        assert _rel(a, b) < 1e-5  # (FP32 atomics of the adjoints in two orders)
    ctx.close()
