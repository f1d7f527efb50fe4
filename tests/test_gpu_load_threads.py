"""Loads from several threads at once: contexts of different lattices, whose
counting kernels need different amounts of shared memory."""
import threading

import numpy as np
import pytest

from tests.helpers import small_case

pytestmark = pytest.mark.gpu


def test_contexts_of_other_sizes_load_at_the_same_time(cuda):
    import latfield2_b200 as L
    errors, start = [], threading.Barrier(4)

    def work(n, npart, seed):
        try:
            cell, off, vel = small_case(n, npart, seed=seed)
            ctx = L.Context(n, box=tuple(v / n[0] for v in n), mode=L.DEPOSIT_FIXED64)
            start.wait(60)
            for _ in range(150):
                ctx.set_particles(cell, off, vel, global_mass=1.0)
            assert ctx.count() == npart and ctx.flags() == 0
            got = ctx.get_particles()["cell"]
            assert np.array_equal(np.sort(got), np.sort(cell))
            ctx.close()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))
            start.abort()
    # 8, 64, 8192 and 32,768 bricks: 32 bytes to 128 KB of counters
    threads = [threading.Thread(target=work, args=a) for a in
               (((32, 32, 32), 500, 1), ((64, 64, 64), 900, 2), ((256, 256, 512), 700, 3),
                ((512, 512, 512), 1000, 4))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors, errors
