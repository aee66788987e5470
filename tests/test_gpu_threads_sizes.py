"""Contexts of different sizes that evaluate at the same time from their own threads.

1100 and 2300 waters at k_max 19 launch the same dipole-step kernels with different amounts of
shared memory above 48 KB (53 and 65 KB); from the host-driven loop they are launched step by step.
Every evaluation gives what the context gives alone, to the order of atomic additions (1e-12, as
in test_gpu_dipole_forms)."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

pytestmark = pytest.mark.gpu


def test_induction_of_two_sizes(product):
    m = Model(data_dir("fs3"))
    sizes = ((1100, 32.05), (2300, 40.98))

    def work(nm, L, reps):
        b = water_box(m, nm, L, 40 + nm, ld=28)
        res = []
        with Context(m, nm, L, precision="fp64") as c:
            c.set_option("graph_loop", 0)
            c.set_ewald(0.35, 19, 19, 19)
            for _ in range(reps):
                out = [np.zeros_like(b.xs) for _ in range(6)]
                e, it = c.nb_induction(b.x, b.y, b.z, b.xs, b.ys, b.zs, L, *out, np.zeros(1))
                assert c.get_option("dipole_row_form_active") == 1
                res.append((e, it))
        return res

    ref = [work(*s, 1)[0] for s in sizes]
    jobs = [(0, 200), (1, 100)] * 4
    with ThreadPoolExecutor(len(jobs)) as pool:
        for (k, _), out in zip(jobs, pool.map(lambda j: work(*sizes[j[0]], j[1]), jobs)):
            for e, it in out:
                assert it == ref[k][1]
                assert abs(e - ref[k][0]) <= 1e-12 * abs(ref[k][0])


def test_reciprocal_sums_of_two_kmax(product):
    """The same for the sums k-vector by k-vector, at k_max 20 and 24 (70 and 82 KB)."""
    m = Model(data_dir("fs3"))
    b = water_box(m, 37, 10.37, 9, ld=28)

    def work(k, reps):
        res = []
        with Context(m, b.nm, b.box, precision="fp64") as c:
            for _ in range(reps):
                f = [np.zeros_like(b.xs) for _ in range(3)]
                res.append(c.kspace_ewald(b.x, b.y, b.z, b.xs, b.ys, b.zs, k, k, k, 0.4, b.box, *f,
                                          np.zeros(1)))
        return res

    ref = {k: work(k, 1)[0] for k in (20, 24)}
    jobs = [20, 24] * 4
    with ThreadPoolExecutor(len(jobs)) as pool:
        for k, out in zip(jobs, pool.map(lambda k: work(k, 1500), jobs)):
            assert max(abs(e - ref[k]) for e in out) <= 1e-12 * abs(ref[k])
