"""The dipole solve of small boxes as one thread-block cluster against the same solve driven
from the host step by step (the row form's step kernels): same iteration count, dipoles, forces
and energy.

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


def _solve(m, b, graph, maxit=None):
    out = [np.zeros_like(b.xs) for _ in range(6)]
    vir = np.zeros(1)
    with Context(m, b.nm, b.box, precision="fp64") as c:
        c.set_option("graph_loop", graph)
        if maxit is not None:
            c.set_maxit(maxit)
        err = None
        try:
            e, it = c.nb_induction(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box, *out, vir)
        except CcpError as ex:
            e, it, err = 0.0, -1, str(ex)
        active = c.get_option("dipole_cluster_active")
    return active, err, e, it, np.stack(out[:3]), np.stack(out[3:]), vir[0]


# one molecule; one site tile per block, some blocks without sites or rows; 128 sites (8 per
# block, none spare) and one molecule more (16 per block, two tiles); a box too large for the form
@pytest.mark.parametrize("nm,L,cluster", [(1, 9.0, 1), (5, 9.0, 1), (16, 7.9, 1), (37, 10.37, 1),
                                          (42, 10.8, 1), (43, 10.88, 1), (128, 15.64, 0)])
def test_cluster_matches_steps(product, nm, L, cluster):
    m = Model(data_dir("fs3"))
    b = water_box(m, nm, L, 300 + nm, ld=28)
    active, err, e, it, mu, F, vir = _solve(m, b, 1)
    assert active == cluster and err is None
    a0, err0, e0, it0, mu0, F0, vir0 = _solve(m, b, 0)
    assert a0 == 0 and err0 is None
    assert it == it0
    assert abs(e - e0) <= TOL * abs(e0)
    assert rel(mu, mu0) <= TOL
    assert rel(F, F0) <= TOL
    assert abs(vir - vir0) <= TOL * abs(vir0)


@pytest.mark.parametrize("maxit", [1, 2, 5])
def test_cluster_stops_at_maxit(product, maxit):
    m = Model(data_dir("fs3"))
    b = water_box(m, 37, 10.37, 9, ld=28)
    r1, r0 = _solve(m, b, 1, maxit), _solve(m, b, 0, maxit)
    assert r1[0] == 1 and r0[0] == 0
    assert r1[1] is not None and r1[1] == r0[1]  # the same report of non-convergence
