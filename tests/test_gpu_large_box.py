"""Boxes at the upper end of what the kernels' shared memory takes.

Both sides of a comparison add the same terms in different orders; a structure factor of n sites
differs by about sqrt(n) * 1.1e-16 of one term's size times sqrt(n), its own size, and the forces
and dipoles by a few times that of their norm (n = 50,000); 1e-12 leaves room for cancellation."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-12


def test_dipole_rows_of_many_sites(product):
    """Five n tiles and more sites than one block's shared memory takes at the few waves of blocks
    that smaller boxes get: the step kernels by rows against those on the factor tables."""
    m = Model(data_dir("fs3"))
    nm = 16640
    b = water_box(m, nm, 79.27, 5, ld=28)
    res = []
    for rows in (1, 0):
        out = [np.zeros_like(b.xs) for _ in range(6)]
        vir = np.zeros(1)
        with Context(m, nm, b.box, precision="fp64") as c:
            c.set_option("dipole_row_form", rows)
            c.set_ewald(0.35, 19, 19, 19)
            e, it = c.nb_induction(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box, *out, vir)
            assert c.get_option("dipole_row_form_active") == rows
        res.append((e, it, np.stack(out[:3]), np.stack(out[3:]), vir[0]))
    (e, it, mu, F, vir), (e0, it0, mu0, F0, vir0) = res
    assert it == it0
    assert abs(e - e0) <= TOL * abs(e0)
    assert rel(mu, mu0) <= TOL
    assert rel(F, F0) <= TOL
    assert abs(vir - vir0) <= TOL * max(abs(vir0), abs(e0))
