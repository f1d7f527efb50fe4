"""Stores with few particles: one, a handful, one below the number of bricks,
where the shares and means that plans are made from round to zero.  The
fixed-point fields are bit-exact against the oracle, the FP32 ones within 1e-6
of FP64 (1e-5 without compensation), in every projection, and with the density
of a step."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import by_id, precision, small_case
from tests.test_gpu_precision import KINDS, _ctx, _fp64

pytestmark = pytest.mark.gpu

N = (64, 64, 64)  # 64 bricks


@pytest.mark.parametrize("npart", [1, 3, 10, 63, 64, 1000])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_deposits_of_few_particles(cuda, npart, mode):
    cell, off, vel = small_case(N, npart, seed=npart, vel_sigma=0.2)
    gm = 1.0 / npart
    ctx = _ctx(N, mode)
    ctx.set_particles(cell, off, vel, global_mass=gm)
    for kind in range(5):
        name, comps = ("deposit_scalar", 1) if kind == 0 else KINDS[kind][:2]
        f = ctx.field(comps)
        getattr(ctx, name)(f)
        got = f.export_internal()
        if mode == 1 and kind:
            acc, e = O.state_deposit_fixed_kind(kind, N, cell, off, vel)
            np.testing.assert_array_equal(got, O.fixed_kind_to_f32(acc, kind, e, gm, 1.0 / N[0]))
            continue
        if mode == 1:
            scale = np.float32(2.0 ** -32 * gm / (1.0 / N[0]) ** 3)
            np.testing.assert_array_equal(got.reshape(-1),
                                          O.fixed_to_f32(O.state_deposit_fixed(N, cell, off), scale))
            continue
        ref, mag = _fp64(N, kind, cell, off, vel, gm)
        for c in range(comps):
            p = precision(got[c], ref[c], mag[c])
            assert p["norm_max"] <= (1e-5 if mode == 2 else 1e-6), (kind, c, p)
            assert mode == 2 or p["cell_max"] <= 1e-6, (kind, c, p)
    assert ctx.flags() == 0
    ctx.close()


@pytest.mark.parametrize("npart", [1, 63, 1000])
@pytest.mark.parametrize("separate", [False, True])
def test_steps_of_few_particles(cuda, npart, separate):
    """A step and the separate calls, the density bit-exact for the particles
    that the context gives back, and those the same as the oracle's."""
    cell, off, vel = small_case(N, npart, seed=npart, vel_sigma=0.05)
    gm = 1.0 / npart
    ctx = _ctx(N, 1)
    ctx.set_particles(cell, off, vel, ids=np.arange(npart, dtype=np.int64), global_mass=gm)
    import torch
    f = np.random.default_rng(2).standard_normal((3, N[2], N[1], N[0])).astype(np.float32)
    F, rho = ctx.field(3, torch.from_numpy(f).cuda()), ctx.field(1)
    if separate:
        ctx.gather_kick(F, 0.05)
        ctx.drift_rebin(0.3)
        ctx.deposit_scalar(rho)
    else:
        ctx.step(F, 0.05, 0.3, rho)
    s = by_id(ctx.get_particles(ids=True))
    v = O.state_kick(N, cell, off, vel, f, np.float32(0.05))
    c, o, _ = O.state_drift(N, cell, off, v, np.float32(0.3 * N[0]))
    for got, want in ((s["cell"], c), (s["off"], o), (s["vel"], v)):
        np.testing.assert_array_equal(got, want)
    scale = np.float32(2.0 ** -32 * gm / (1.0 / N[0]) ** 3)
    np.testing.assert_array_equal(rho.export_internal().reshape(-1),
                                  O.fixed_to_f32(O.state_deposit_fixed(N, c, o), scale))
    assert ctx.flags() & ~0x8 == 0
    ctx.close()
