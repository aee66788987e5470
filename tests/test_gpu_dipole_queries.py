"""The queries that tell which form the last dipole solve ran in."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Context, Model, _lib, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

pytestmark = pytest.mark.gpu


def test_cluster_query_tells_of_the_last_solve(product):
    """37 waters: one cluster, except beside FS3's gradients by triples and from the host."""
    import torch
    m = Model(data_dir("fs3"))
    b = water_box(m, 37, 10.37, 9)
    args = [torch.as_tensor(np.ascontiguousarray(getattr(b, k)), device="cuda")
            for k in ("x", "y", "z", "xs", "ys", "zs")]
    with Context(m, b.nm, b.box) as c:
        assert c.get_option("dipole_cluster_active") == 0
        for opts, active in (({}, 1), ({"fs3_param_grad": 1}, 0), ({"fs3_param_grad": 0}, 1),
                             ({"graph_loop": 0}, 0), ({"graph_loop": 1}, 1)):
            for k, v in opts.items():
                c.set_option(k, v)
            c.terms_device(_lib.TERM_INDUCTION | _lib.TERM_FS3, *args, b.box)
            assert c.get_option("dipole_cluster_active") == active, opts
            assert c.get_option("dipole_grid_active") == 0
