"""A wait between the blocks of the one-grid dipole solve that runs out: the kernel leaves with its
error state, and the evaluation is repeated with the step kernels.  The limit of one poll makes
every first wait run out.

The step kernels' results equal those of the same kernels driven from the host to the rounding of
their sums (test_gpu_dipole_forms derives 1e-12)."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import CcpError, Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("solver", [0, 1])
def test_wait_that_runs_out(product, solver):
    m = Model(data_dir("fs2fs3"))
    b = water_box(m, 128, 15.64, 31, ld=28)

    def hot(c):
        r = c.hot_path(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box)
        return (r.energies, np.stack([r.idmx, r.idmy, r.idmz]), np.stack([r.fxs, r.fys, r.fzs]))

    with Context(m, b.nm, b.box, precision="fp64") as c:
        c.set_option("dipole_solver", solver)
        with pytest.raises(CcpError, match="positive"):
            c.set_option("dipole_grid_polls", 0)
        polls = c.get_option("dipole_grid_polls")
        c.set_option("graph_loop", 0)
        e0, mu0, f0 = hot(c)
        c.set_option("graph_loop", 1)

        def check(active):
            e, mu, f = hot(c)
            assert c.get_option("dipole_grid_active") == active
            assert e["ind_iters"] == e0["ind_iters"]
            for k in ("scpe", "rcpe", "kcpe", "indpe", "fs2pe", "fs3pe", "vir"):
                assert abs(e[k] - e0[k]) <= TOL * abs(e0[k]), k
            assert rel(mu, mu0) <= TOL
            assert rel(f, f0) <= TOL

        check(1)
        c.set_option("dipole_grid_polls", 1)
        check(0)  # runs out, is repeated
        c.set_option("dipole_grid_polls", 1)
        check(0)  # the same from a context whose buffers hold a solve
        check(0)  # stays with the step kernels
        c.set_option("dipole_grid_polls", polls)
        check(1)
