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


def test_fs3_with_the_longest_neighbour_lists(product, tmp_path):
    """A cut-off radius that makes all of 7300 molecules neighbours: longer lists than the pair
    form's shared memory takes, not longer than the triple form's.  FS3 runs, by triples, and gives
    what the ordinary cut-off radius gives, which FS3 does not depend on (by pairs; both add the
    same terms in different orders, test_gpu_fs3_pairs derives 1e-10)."""
    nm, L = 7300, 60.23
    for p in data_dir("fs3").iterdir():
        t = p.read_text()
        if p.name == "CONTROL":
            assert t.count("9.0                 # rcut ") == 1
            t = t.replace("9.0                 # rcut ", "53.0                # rcut ")
        (tmp_path / p.name).write_text(t)
    m0, m1 = Model(data_dir("fs3")), Model(tmp_path)
    b = water_box(m0, nm, L, 6, ld=28)
    res = []
    for m, active in ((m1, 0), (m0, 1)):
        f = [np.zeros_like(b.xs) for _ in range(3)]
        c2, c3 = ([np.zeros(nm) for _ in range(3)] for _ in range(2))
        vir = np.zeros(1)
        with Context(m, nm, L, precision="fp64") as c:
            e2, e3 = c.threebody_term(b.x, b.y, b.z, b.xs, b.ys, b.zs, L, *f, *c2, *c3, vir)
            assert c.get_option("fs3_pair_form_active") == active
        res.append((e3, np.stack(f), np.stack(c3), vir[0]))
    (e, f, c3, vir), (e0, f0, c0, vir0) = res
    assert abs(e - e0) <= 1e-10 * abs(e0)
    assert rel(f, f0) <= 1e-10
    assert rel(c3, c0) <= 1e-10
    assert abs(vir - vir0) <= 1e-10 * abs(vir0)
