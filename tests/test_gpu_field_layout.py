"""Field import and export in the reference's layout (interleaved components,
halo) against numpy, for the component counts with kernels of their own and
others, rows of one site to several chunks (by sites below 48, by rows above), and halos up to the lattice."""
import numpy as np
import pytest

from tests.helpers import internal_to_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,halo", [((5, 6, 7), 0), ((5, 6, 7), 5), ((33, 4, 9), 1), ((70, 3, 2), 2),
                                    ((1, 1, 40), 1), ((700, 1, 1), 0), ((513, 2, 1), 1),
                                    ((2, 3, 50), 0), ((47, 3, 5), 0), ((16, 2, 2), 16),
                                    ((5000, 1, 1), 0)])
@pytest.mark.parametrize("comps", [1, 2, 3, 6, 7])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_import_and_export(cuda, n, halo, comps, dtype):
    import latfield2_b200 as L
    ctx = L.Context(n, box=tuple(v / n[0] for v in n))
    rng = np.random.default_rng(comps)
    A = rng.standard_normal((comps, n[2], n[1], n[0])).astype(np.float32)
    ref = internal_to_reference(A, halo).astype(dtype)
    ref_garbage = ref.copy()  # the halo is not read
    if halo:
        ref_garbage[:halo] = 7.0
    f = ctx.field(comps)
    f.import_(ref_garbage, halo=halo)
    np.testing.assert_array_equal(f.export_internal(), A)
    np.testing.assert_array_equal(f.export(halo, dtype, fill_halo=True), ref)
    out = f.export(halo, dtype)
    inner = tuple(slice(halo, halo + m) for m in (n[2], n[1], n[0]))
    np.testing.assert_array_equal(out[inner], ref[inner])
    out[inner] = 0
    assert not out.any()
