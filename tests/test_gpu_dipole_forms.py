"""The dipole solve as one thread-block cluster (small boxes) and as one cooperative grid (middle
sizes) against the same solve driven from the host step by step (the row form's step kernels):
same iteration count, dipoles, forces and energy.

Both add the same terms in a different order.  A step's field then differs by some
sqrt(n) * 1.1e-16 of its size (n < 2000 terms per component), and the solve contracts the
differences of earlier steps, so the converged dipoles agree to about 1e-14; 1e-12 leaves room
for cancellation in the small ones.
"""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import CcpError, Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _solve(m, b, graph, maxit=None, solver=0):
    out = [np.zeros_like(b.xs) for _ in range(6)]
    vir = np.zeros(1)
    with Context(m, b.nm, b.box, precision="fp64") as c:
        c.set_option("graph_loop", graph)
        c.set_option("dipole_solver", solver)
        if maxit is not None:
            c.set_maxit(maxit)
        err = None
        try:
            e, it = c.nb_induction(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box, *out, vir)
        except CcpError as ex:
            e, it, err = 0.0, -1, str(ex)
        active = c.get_option("dipole_cluster_active") + 2 * c.get_option("dipole_grid_active")
    return active, err, e, it, np.stack(out[:3]), np.stack(out[3:]), vir[0]


CLUSTER, GRID = 1, 2


# one molecule; one site tile per block, some blocks without sites or rows; 128 sites (8 per
# block, none spare) and one molecule more (16 per block, two tiles); a box too large for the form
@pytest.mark.parametrize("nm,L,cluster", [(1, 9.0, 1), (5, 9.0, 1), (16, 7.9, 1), (37, 10.37, 1),
                                          (42, 10.8, 1), (43, 10.88, 1)])
def test_cluster_matches_steps(product, nm, L, cluster):
    _compare(nm, L, cluster, 0)


def _compare(nm, L, form, solver):
    m = Model(data_dir("fs3"))
    b = water_box(m, nm, L, 300 + nm, ld=28)
    active, err, e, it, mu, F, vir = _solve(m, b, 1, solver=solver)
    assert active == form and err is None
    a0, err0, e0, it0, mu0, F0, vir0 = _solve(m, b, 0, solver=solver)
    assert a0 == 0 and err0 is None
    assert it == it0
    assert abs(e - e0) <= TOL * abs(e0)
    assert rel(mu, mu0) <= TOL
    assert rel(F, F0) <= TOL
    assert abs(vir - vir0) <= TOL * abs(vir0)


# blocks of 8 sites with the last ones short; one molecule more than one per block of 8 sites;
# 9 to 16 sites per block (two tiles), an odd number of them; three tiles; with one to several
# operand chunks per block, resident or through the ring
@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("nm,L", [(65, 12.5), (128, 15.64), (394, 22.8), (395, 22.8), (601, 26.2),
                                  (903, 30.0)])
def test_grid_matches_steps(product, nm, L, solver):
    _compare(nm, L, GRID, solver)


@pytest.mark.parametrize("nm,L,form,solver", [(37, 10.37, CLUSTER, 0), (128, 15.64, GRID, 0),
                                              (128, 15.64, GRID, 1)])
@pytest.mark.parametrize("maxit", [1, 2, 5])
def test_stops_at_maxit(product, maxit, nm, L, form, solver):
    m = Model(data_dir("fs3"))
    b = water_box(m, nm, L, 9, ld=28)
    r1, r0 = _solve(m, b, 1, maxit, solver), _solve(m, b, 0, maxit, solver)
    assert r1[0] == form and r0[0] == 0
    assert r1[1] is not None and r1[1] == r0[1]  # the same report of non-convergence


def test_grid_from_several_threads(product):
    """Contexts of several threads evaluate at the same time: at most one at a time takes the
    grid form, the others the step kernels, and all get the same results."""
    from concurrent.futures import ThreadPoolExecutor

    m = Model(data_dir("fs3"))
    b = water_box(m, 128, 15.64, 1001, ld=28)
    ref = _solve(m, b, 0)
    with ThreadPoolExecutor(4) as pool:
        res = list(pool.map(lambda _: _solve(m, b, 1), range(16)))
    for r in res:
        assert r[1] is None and r[3] == ref[3]
        assert abs(r[2] - ref[2]) <= TOL * abs(ref[2])
        assert rel(r[4], ref[4]) <= TOL and rel(r[5], ref[5]) <= TOL
