"""When the dipole steps take the full phase matrix, and that the choice does not change results.

The forms add the same products of the same phases in different orders (test_gpu_krows derives
1e-12 for sums of up to 1000 sites)."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-12


# past the row form's k_max, where the matrix fits in half of the L2 and where it does not (128
# waters: 104 MB); within it, with the row form and without
@pytest.mark.parametrize("nm,L,k,rows,active", [(37, 10.37, 20, 1, 1), (64, 12.42, 20, 1, 1),
                                                (128, 15.64, 20, 1, 0), (37, 10.37, 13, 1, 0),
                                                (37, 10.37, 13, 0, 1)])
def test_default_takes_the_matrix_without_rows(product, nm, L, k, rows, active):
    m = Model(data_dir("fs3"))
    b = water_box(m, nm, L, 800 + nm, ld=28)
    res = []
    for full in (None, 0):
        out = [np.zeros_like(b.xs) for _ in range(6)]
        vir = np.zeros(1)
        with Context(m, nm, b.box, precision="fp64") as c:
            c.set_option("dipole_row_form", rows)
            if full is not None:
                c.set_option("phase_matrix_full", full)
            c.set_ewald(0.35, k, k, k)
            e, it = c.nb_induction(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box, *out, vir)
            assert c.get_option("phase_matrix_full_active") == (active if full is None else 0)
        res.append((e, it, np.stack(out[:3]), np.stack(out[3:]), vir[0]))
    (e, it, mu, F, vir), (e0, it0, mu0, F0, vir0) = res
    assert it == it0
    assert abs(e - e0) <= TOL * abs(e0)
    assert rel(mu, mu0) <= TOL
    assert rel(F, F0) <= TOL
    assert abs(vir - vir0) <= TOL * max(abs(vir0), abs(e0))
