"""FS3 by molecule pairs against FS3 by triples (option fs3_pair_form = 0): energy, counts, site
and COM forces, virial and parameter gradients.

Both add the same terms: a triple's energy sums some 5000 products of both signs that cancel to
between 1e-2 and 1e-4 of their size, so two orders of summation differ by about
sqrt(5000) * 1.1e-16 * 1e4 = 1e-10 of a triple's energy at worst, and less of the totals, where
the triples' rounding averages out.  1e-10 is the bound, the FP64 parity tests' one."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _run(m, b, pair, grad):
    f = [np.zeros_like(b.xs) for _ in range(3)]
    c2, c3 = ([np.zeros(b.nm) for _ in range(3)] for _ in range(2))
    vir = np.zeros(1)
    with Context(m, b.nm, b.box, precision="fp64") as c:
        c.set_option("fs3_pair_form", pair)
        c.set_option("fs3_param_grad", int(grad))
        e = [c.threebody_term(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box, *f, *c2, *c3, vir)]
        active = c.get_option("fs3_pair_form_active")
        # once more on the buffers that the first evaluation grew
        for a in f + c2 + c3:
            a[:] = 0.0
        vir[:] = 0.0
        e.append(c.threebody_term(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box, *f, *c2, *c3, vir))
        g = c.fs3_param_grad() if grad else ()
    assert abs(e[0][1] - e[1][1]) <= 1e-12 * abs(e[0][1])
    return active, e[1][1], np.stack(f), np.stack(c3), vir[0], g


# no triple; one triple at most; a box just wider than two cut-offs, sparse and dense (the visit
# lists and pairs outgrow their first sizes); ordinary sizes, ragged ones among them
@pytest.mark.parametrize("nm,L", [(2, 20.0), (3, 13.0), (20, 12.65), (67, 12.65), (100, 12.65),
                                  (128, 15.64), (201, 18.2), (333, 21.5)])
def test_pairs_match_triples(product, nm, L):
    m = Model(data_dir("fs3"))
    b = water_box(m, nm, L, 600 + nm, ld=28, min_oo=2.2 if nm == 100 else 2.5)
    a1, e1, f1, c1, v1, _ = _run(m, b, 1, False)
    a0, e0, f0, c0, v0, _ = _run(m, b, 0, False)
    assert (a1, a0) == (1, 0)
    assert abs(e1 - e0) <= TOL * abs(e0)
    assert rel(f1, f0) <= TOL
    assert rel(c1, c0) <= TOL
    assert abs(v1 - v0) <= TOL * abs(v0)


@pytest.mark.parametrize("nm,L", [(3, 13.0), (67, 12.65), (128, 15.64), (201, 18.2)])
def test_parameter_gradients(product, nm, L):
    m = Model(data_dir("fs3"))
    b = water_box(m, nm, L, 700 + nm, ld=28)
    a1, e1, f1, c1, v1, g1 = _run(m, b, 1, True)
    a0, e0, f0, c0, v0, g0 = _run(m, b, 0, True)
    assert (a1, a0) == (1, 0)
    assert abs(e1 - e0) <= TOL * abs(e0)
    assert rel(f1, f0) <= TOL
    for x, y in zip(g1, g0):
        assert rel(x, y) <= TOL


def test_small_box_takes_triples(product):
    """Up to two cut-offs a triple's molecules can be neighbours by more than one image."""
    m = Model(data_dir("fs3"))
    b = water_box(m, 60, 12.55, 9, ld=28)
    assert _run(m, b, 1, False)[0] == 0
