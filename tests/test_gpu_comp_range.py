"""The compensated FP32 mode over the range of units: masses and velocities
scaled by powers of two give the field scaled by the product's power, wherever
the terms are normal FP32 numbers, whether the sums are integers in a common
unit or the FP32 pairs that hold anything."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import positions, precision
from tests.test_gpu_precision import KINDS, _fp64

pytestmark = pytest.mark.gpu

N = (8, 8, 8)
NPART = 400


def _case():
    """Offsets in [1/4, 3/4], masses and |v_i| in [1/2, 1): a term is at least
    2^-9 of the largest."""
    rng = np.random.default_rng(3)
    cell = rng.integers(0, 512, NPART).astype(np.int32)
    off = (0.25 + 0.5 * rng.random((NPART, 3))).astype(np.float32)
    vel = ((0.5 + 0.49 * rng.random((NPART, 3))) * rng.choice([-1, 1], (NPART, 3))).astype(np.float32)
    mass = (0.5 + 0.49 * rng.random(NPART)).astype(np.float32)
    return cell, off, vel, mass


@pytest.mark.parametrize("individual", [False, True])
@pytest.mark.parametrize("kind", [0, 1, 2, 3, 4])
def test_units_of_mass_and_velocity(cuda, kind, individual):
    import latfield2_b200 as L
    cell, off, vel, mass = _case()
    power = (0, 1, 2, 1, 2)[kind]
    if individual:  # FP64 reference: the projection of the masses' multiples
        cs, order = O.lists_from_insertion(N, cell)
        pos = positions(N, 1.0, cell, off)[order]
        if kind == 0:
            ref = O.state_deposit_f64(N, cell, off, 1.0, mass=mass).reshape(1, *N)
            mag = ref
        else:
            ref, mag = (O.interior(KINDS[kind][2](N, 1, 1.0, cs, pos, v.astype(np.float64)[order],
                                                  pmass=mass.astype(np.float64)[order]), N, 1)
                        for v in (vel, np.abs(vel)))
    else:
        ref, mag = _fp64(N, kind, cell, off, vel, 8.0 ** -3)
    ctx = L.Context(N, box=8.0 if individual else 1.0, mode=L.DEPOSIT_FP32)
    name, comps = ("deposit_scalar", 1) if kind == 0 else KINDS[kind][:2]
    f = ctx.field(comps)
    tried = 0
    for em in list(range(-100, 101, 20)) + [-83, -44, -91, 91]:
        for ev in (-45, -41, -35, -34, -17, 0, 17, 39, 41, 45) if power else (0,):
            k = em + power * ev
            # every term and every partial product a normal number, the sums finite
            if not (-117 <= k <= 110 and -117 <= em + ev <= 110):
                continue
            s = 2.0 ** em
            ctx.set_particles(cell, off, np.ldexp(vel, ev).astype(np.float32),
                              mass=(mass * np.float32(s)) if individual else None,
                              global_mass=0.0 if individual else s * 8.0 ** -3)
            getattr(ctx, name)(f)
            got = np.ldexp(f.export_internal().astype(np.float64), -k)
            for c in range(comps):
                p = precision(got[c], ref[c], mag[c])
                assert p["norm_max"] <= 1e-6 and p["cell_max"] <= 1e-6, (em, ev, c, p)
            tried += 1
    assert tried >= (11 if power == 0 else 40)
    assert ctx.flags() == 0
    ctx.close()


def _wide_case(name, npart=6000, n=(20, 20, 20)):
    """Terms far below the largest of their brick, whole vertices among them."""
    rng = np.random.default_rng(11)
    cell = rng.integers(0, n[0] * n[1] * n[2], npart).astype(np.int32)
    off = (rng.random((npart, 3)) * (1 - 2.0 ** -23)).astype(np.float32)
    vel = rng.standard_normal((npart, 3)).astype(np.float32)
    mass = np.full(npart, 1.0 / npart, np.float32)
    few = rng.choice(npart, 60, replace=False)
    if name == "fast one":  # a slow population beside one fast particle per brick
        vel *= np.float32(1e-6)
        vel[few[:8]] = (0.9, -0.7, 0.8)
    elif name == "slow few":  # few enough for the list of rests
        vel[few] *= np.float32(1e-9)
    elif name == "planar":  # every T_i2 term far below T_00
        vel[:, 2] *= np.float32(1e-9)
    elif name == "light few":
        mass[few] *= np.float32(1e-20)
        cell[few] = np.arange(60) * 133
    else:
        assert name == "light"
        mass = (10.0 ** rng.uniform(-25, 0, npart)).astype(np.float32)
    return n, cell, off, vel, mass


@pytest.mark.parametrize("name", ["fast one", "slow few", "planar", "light few", "light"])
@pytest.mark.parametrize("kind", [0, 1, 2, 3, 4])
def test_small_terms_beside_large_ones(cuda, kind, name):
    """Every vertex that a particle touches, however small its sum beside the
    others': within 1e-6 of the sum of its |terms| (six FP32 roundings of
    2^-24 at most, the sum being exact)."""
    import latfield2_b200 as L
    n, cell, off, vel, mass = _wide_case(name)
    res = 1.0 / n[0]
    if kind == 0:
        ref = O.state_deposit_f64(n, cell, off, res, mass=mass).reshape(1, *n)
        mag = ref
    else:
        cs, order = O.lists_from_insertion(n, cell)
        pos = positions(n, res, cell, off)[order]
        ref, mag = (O.interior(KINDS[kind][2](n, 1, res, cs, pos, v.astype(np.float64)[order],
                                              pmass=mass.astype(np.float64)[order]), n, 1)
                    for v in (vel, np.abs(vel)))
    ctx = L.Context(n, box=1.0, mode=L.DEPOSIT_FP32)
    ctx.set_particles(cell, off, vel, mass=mass)
    f = ctx.field(ref.shape[0])
    getattr(ctx, ("deposit_scalar" if kind == 0 else KINDS[kind][0]))(f)
    got = f.export_internal()
    for c in range(ref.shape[0]):
        some = mag[c] > 0
        err = np.abs(got[c].astype(np.float64) - ref[c])[some] / mag[c][some]
        assert err.max() <= 1e-6, (c, err.max())
        assert not got[c][~some].any()
    ctx.close()


def test_single_terms_are_exact(cuda):
    """A vertex that one term reaches holds that term, at every power of two
    below the brick's largest and for values of 24 bits."""
    import latfield2_b200 as L
    n = (32, 32, 32)
    k = np.arange(120)
    cell = np.array([(2 * i % 16) + 32 * ((2 * i // 16 * 2) % 16) + 1024 * (2 * (i // 64)) for i in k],
                    np.int32)
    assert len(set(cell)) == 120
    mass = (np.ldexp(1.0, -(k // 2)) * np.where(k % 2, 1.0, 1.0 - 2.0 ** -24)).astype(np.float32)
    ctx = L.Context(n, box=32.0, mode=L.DEPOSIT_FP32)
    ctx.set_particles(cell, np.zeros((120, 3), np.float32), np.zeros((120, 3), np.float32), mass=mass)
    f = ctx.field(1)
    ctx.deposit_scalar(f)
    got = f.export_internal().reshape(-1)
    np.testing.assert_array_equal(got[cell], mass)
    ctx.close()


@pytest.mark.parametrize("name", ["light few", "light"])
def test_chain_deposit_of_light_particles(cuda, name):
    """The brick-tiled deposit of the chain: every vertex within the roundings
    of its terms (three each) and of the FP32 additions to the field (a rest or
    a brick's sum each, under 30 here), 2^-24 of the sum apiece."""
    import torch
    import latfield2_b200 as L
    from latfield2_b200.autodiff import _Ops
    n, cell, off, _, mass = _wide_case(name)
    xyz = np.stack([cell % n[0], cell // n[0] % n[1], cell // (n[0] * n[1])], 1)
    nb = [(m + 15) // 16 for m in n]
    brick = xyz[:, 0] // 16 + nb[0] * (xyz[:, 1] // 16 + nb[1] * (xyz[:, 2] // 16))
    order = np.lexsort((cell, brick))
    c, o, m = (torch.from_numpy(a[order]).cuda() for a in (cell, off, mass))
    ctx = L.Context(n, box=1.0, mode=L.DEPOSIT_FP32)
    ops = _Ops(ctx)
    ops.bricks = ops.brick_start(c)
    rho = torch.zeros(n[0] * n[1] * n[2], device="cuda")
    ops.deposit(c, o, m, rho)
    ref = O.state_deposit_f64(n, cell, off, 1.0 / n[0], mass=mass)
    some = ref > 0
    got = rho.cpu().numpy()
    assert (np.abs(got.astype(np.float64) - ref)[some] / ref[some]).max() <= 33 * 2.0 ** -24
    assert not got[~some].any()
    ctx.close()
