"""Deposits of bricks that are split over several CTAs (parts of heavy
bricks): bricks one particle below and above the threshold, a brick of
tens of parts beside empty ones, on a lattice of whole bricks and on a ragged
one.  The fixed-point fields are bit-exact against the oracle; the FP32 modes
are within the tolerances of test_gpu_precision.py (1e-6 compensated, 1e-5 of
the field maximum for unordered FP32 sums)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import by_id, precision, small_case
from tests.test_gpu_precision import KINDS, _ctx, _deposit, _fp64

pytestmark = pytest.mark.gpu


def _in_brick(n, brick, count, seed):
    """`count` particles anywhere in the cells of one brick."""
    rng = np.random.default_rng(seed)
    ext = [min(16, n[d] - 16 * brick[d]) for d in range(3)]
    xyz = [16 * brick[d] + rng.integers(0, ext[d], count) for d in range(3)]
    cell = (xyz[0] + n[0] * (xyz[1] + n[1] * xyz[2])).astype(np.int32)
    off = (rng.random((count, 3)) * (1 - 2.0 ** -23)).astype(np.float32)
    vel = (0.2 * rng.standard_normal((count, 3))).astype(np.float32)
    return cell, off, vel


def _case(name):
    # parts of 4096 particles: bricks above 6144 are split
    if name == "edges":
        n = (64, 32, 48)
        bits = [_in_brick(n, (0, 0, 0), 6144, 1), _in_brick(n, (3, 1, 2), 6145, 2),
                _in_brick(n, (1, 1, 1), 8193, 3), _in_brick(n, (2, 0, 1), 1, 4)]
    else:
        n = (33, 17, 24)
        bits = [_in_brick(n, (1, 0, 0), 30011, 5), _in_brick(n, (2, 1, 1), 9000, 6),
                small_case(n, 500, seed=7, vel_sigma=0.2)]
    return (n,) + tuple(np.concatenate([b[k] for b in bits]) for k in range(3))


@pytest.mark.parametrize("name", ["edges", "ragged"])
@pytest.mark.parametrize("kind", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_split_bricks(cuda, name, kind, mode):
    n, cell, off, vel = _case(name)
    gm = 1.0 / cell.shape[0]
    got = _deposit(n, mode, kind, cell, off, vel, gm)
    ref, mag = _fp64(n, kind, cell, off, vel, gm)
    for c in range(ref.shape[0]):
        p = precision(got[c], ref[c], mag[c])
        assert p["norm_max"] <= (1e-5 if mode == 2 else 1e-6), (c, p)
        assert mode == 2 or p["cell_max"] <= 1e-6, (c, p)
    if mode == 1 and kind:
        acc, e = O.state_deposit_fixed_kind(kind, n, cell, off, vel)
        np.testing.assert_array_equal(got, O.fixed_kind_to_f32(acc, kind, e, gm, 1.0 / n[0]))
    elif mode == 1:
        scale = np.float32(2.0 ** -32 * gm / (1.0 / n[0]) ** 3)
        np.testing.assert_array_equal(got.reshape(-1),
                                      O.fixed_to_f32(O.state_deposit_fixed(n, cell, off), scale))


@pytest.mark.parametrize("spread", [0.1, 30.0])
@pytest.mark.parametrize("kind", [0, 1, 2, 3, 4])
def test_split_bricks_with_individual_masses(cuda, kind, spread):
    """Masses up to 1.1 or about 20 of their mean: the bound on the particles
    that two 32-bit words sum exactly follows the largest mass of the part."""
    n, cell, off, vel = _case("ragged")
    npart = cell.shape[0]
    u = np.random.default_rng(9).random(npart)
    m = ((1.0 + (spread * (2 * u - 1) if spread < 1 else spread * (u > 0.97))) / npart).astype(np.float32)
    unit = float(np.sum(m.astype(np.float64)) / npart)
    mrel = (m * np.float32(1.0 / unit)).astype(np.float32)
    ctx = _ctx(n, 1)
    ctx.set_particles(cell, off, vel, mass=m)
    name, comps = ("deposit_scalar", 1) if kind == 0 else KINDS[kind][:2]
    f = ctx.field(comps)
    getattr(ctx, name)(f)
    got = f.export_internal()
    if kind == 0:
        scale = np.float32(2.0 ** -32 * unit / (1.0 / n[0]) ** 3)
        want = O.fixed_to_f32(O.state_deposit_fixed(n, cell, off, mrel=mrel), scale).reshape(got.shape)
    else:
        acc, e = O.state_deposit_fixed_kind(kind, n, cell, off, vel, mrel=mrel)
        want = O.fixed_kind_to_f32(acc, kind, e, unit, 1.0 / n[0])
    np.testing.assert_array_equal(got, want)
    ctx.close()


def test_compensated_sums_outside_the_integer_range(cuda):
    """Terms that the compensated mode's integers do not take (a velocity unit
    of 1e-15 squared, masses far from 1, an infinity): the FP32 sums give the
    scaled field, and an infinity or NaN stays at the vertices it reaches."""
    n, cell, off, vel = _case("ragged")
    npart = cell.shape[0]
    gm = 1.0 / npart
    for kind in (2, 4):
        got = _deposit(n, 0, kind, cell, off, vel * np.float32(2.0 ** -50), gm)
        ref, mag = _fp64(n, kind, cell, off, vel, gm)
        for c in range(ref.shape[0]):
            p = precision(got[c].astype(np.float64) * 2.0 ** 100, ref[c], mag[c])
            assert p["norm_max"] <= 1e-6 and p["cell_max"] <= 1e-6, (c, p)
    bad = vel.copy()
    bad[7] = (np.inf, 0.5, 0.25)
    ctx = _ctx(n, 0)
    ctx.set_particles(cell, off, bad, global_mass=gm)
    f = ctx.field(3)
    ctx.deposit_vector_cic(f)
    got = f.export_internal()
    ref, _ = _fp64(n, 3, cell, off, vel, gm)
    ref2, _ = _fp64(n, 3, np.delete(cell, 7), np.delete(off, 7, 0), np.delete(vel, 7, 0), gm)
    touched = np.abs(ref - ref2) > 0
    assert not np.isfinite(got[0][touched[0]]).any()
    assert np.isfinite(got[0][~touched[0]]).all() and np.isfinite(got[1:]).all()
    ctx.close()


def test_compensated_sums_with_a_wide_range_of_masses(cuda):
    """Masses over seven decades in one brick: each vertex to 2e-7 of its sum
    wherever that is above 1e-9 of the largest mass's contribution, the unit
    of the integers being 2^-48 of it."""
    n = (20, 20, 20)
    cell, off, vel = small_case(n, 4000, seed=23, vel_sigma=0.1)
    m = (10.0 ** np.random.default_rng(1).uniform(-7, 0, 4000)).astype(np.float32)
    ctx = _ctx(n, 0)
    ctx.set_particles(cell, off, vel, mass=m)
    f = ctx.field(1)
    ctx.deposit_scalar(f)
    got = f.export_internal()[0].astype(np.float64).reshape(-1)
    ref = O.state_deposit_f64(n, cell, off, 1.0 / 20, mass=m)
    sel = ref > 1e-9 * 8000
    # three FP32 products and the rounding of the sum: 4 ulp of 2^-24
    assert np.max(np.abs(got[sel] - ref[sel]) / ref[sel]) < 4 * 2.0 ** -24 + 8 * 2.0 ** -48 / 1e-9
    ctx.close()


def test_more_bricks_than_a_load_counts_in_shared_memory(cuda):
    """51,201 bricks: the load counts in global memory, the plan of heavy bricks
    and the move's order take several CTAs, and the rebin tail plans the scalar
    deposit.  Bit-exact against the oracle before and after a step."""
    import torch
    n = (2, 2, 16 * 51201)
    rng = np.random.default_rng(6)
    z = np.concatenate([rng.integers(0, n[2], 20000), 16 * 40000 + rng.integers(0, 16, 15000),
                        16 * 51200 + rng.integers(0, 16, 5000)])
    npart = z.size
    cell = (rng.integers(0, 2, npart) + 2 * (rng.integers(0, 2, npart) + 2 * z)).astype(np.int32)
    off = (rng.random((npart, 3)) * (1 - 2.0 ** -23)).astype(np.float32)
    vel = (0.2 * rng.standard_normal((npart, 3))).astype(np.float32)
    gm = 1.0 / npart
    ctx = _ctx(n, 1)
    ctx.set_particles(cell, off, vel, ids=np.arange(npart, dtype=np.int64), global_mass=gm)
    scale = np.float32(2.0 ** -32 * gm / 0.5 ** 3)
    f, v = ctx.field(1), ctx.field(3)

    def check(field, c, o):
        np.testing.assert_array_equal(field.export_internal().reshape(-1),
                                      O.fixed_to_f32(O.state_deposit_fixed(n, c, o), scale))
    ctx.deposit_scalar(f)
    check(f, cell, off)
    ctx.deposit_vector(v)
    acc, e = O.state_deposit_fixed_kind(1, n, cell, off, vel)
    np.testing.assert_array_equal(v.export_internal(), O.fixed_kind_to_f32(acc, 1, e, gm, 0.5))
    F = torch.from_numpy(rng.standard_normal((3, n[2], n[1], n[0])).astype(np.float32)).cuda()
    ctx.step(ctx.field(3, F), 0.05, 0.3, f)
    s = ctx.get_particles(ids=True)
    assert not np.array_equal(by_id(s)["cell"], cell)
    check(f, s["cell"], s["off"])
    assert ctx.flags() & ~0x8 == 0
    ctx.close()


def test_a_store_that_clumps_after_its_load(cuda):
    """An even store deposits without a plan of heavy bricks; one that collapses
    into a brick afterwards is bit-exact whether the host has read its counts
    since (the maximum velocity) or not, after a few steps and after many."""
    import torch
    n = (64, 64, 64)
    rng = np.random.default_rng(12)
    npart = 60000
    cell = rng.integers(0, 64 ** 3, npart).astype(np.int32)
    off = (rng.random((npart, 3)) * (1 - 2.0 ** -23)).astype(np.float32)
    xyz = np.stack([cell % 64, cell // 64 % 64, cell // 4096], 1) + off
    gm = 1.0 / npart
    ctx = _ctx(n, 1)
    # towards the middle of brick (1, 1, 1): nearly all of them there after 8 steps
    vel = ((24.0 - xyz) / 64.0).astype(np.float32)
    ctx.set_particles(cell, off, vel, global_mass=gm)
    F = ctx.field(3, torch.zeros(3, 64, 64, 64, device="cuda"))
    rho, vec = ctx.field(1), ctx.field(3)

    def check(stepped):
        s = ctx.get_particles()
        scale = np.float32(2.0 ** -32 * gm / (1.0 / n[0]) ** 3)
        want = O.fixed_to_f32(O.state_deposit_fixed(n, s["cell"], s["off"]), scale)
        if stepped:
            np.testing.assert_array_equal(rho.export_internal().reshape(-1), want)
        ctx.deposit_scalar(rho)
        np.testing.assert_array_equal(rho.export_internal().reshape(-1), want)
        ctx.deposit_vector(vec)
        acc, e = O.state_deposit_fixed_kind(1, n, s["cell"], s["off"], s["vel"])
        np.testing.assert_array_equal(vec.export_internal(), O.fixed_kind_to_f32(acc, 1, e, gm, 1.0 / n[0]))
        return np.bincount(s["cell"] % 64 // 16 + 4 * (s["cell"] // 64 % 64 // 16)
                           + 16 * (s["cell"] // 4096 // 16)).max()
    assert check(False) < 1200
    for _ in range(8):
        ctx.step(F, 0.0, 0.11, rho)
    assert check(True) > 40000
    ctx.last_max_velocity()
    check(True)
    for _ in range(40):
        ctx.step(F, 0.0, 0.0, rho)
    check(True)
    assert ctx.flags() & ~0x8 == 0
    ctx.close()
