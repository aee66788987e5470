"""Models without charged or without polarisable sites: the sums over no site are refused with an
error, as the launches of no blocks that they would need."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import CcpError, Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

pytestmark = pytest.mark.gpu


def _model(tmp_path, charges, npol):
    for p in data_dir("fs3").iterdir():
        lines = p.read_text().split("\n")
        if p.name == "FIELD":
            assert lines[3].split()[0] == "3"
            lines[3] = lines[3].replace("3", str(npol), 1)
            for k in range(5, 33):  # name, x, y, z, mass, charge, polarizability
                t = lines[k].split()
                if not charges:
                    t[5] = "0.0"
                lines[k] = "  ".join(t)
        (tmp_path / p.name).write_text("\n".join(lines))
    return Model(tmp_path)


def test_reciprocal_sum_without_charges(product, tmp_path):
    b = water_box(Model(data_dir("fs3")), 37, 10.37, 9, ld=28)
    m = _model(tmp_path, charges=False, npol=3)
    f = [np.zeros_like(b.xs) for _ in range(3)]
    with Context(m, b.nm, b.box) as c:
        for _ in range(2):  # the context stays usable
            with pytest.raises(CcpError, match="invalid configuration"):
                c.kspace_ewald(b.x, b.y, b.z, b.xs, b.ys, b.zs, 5, 5, 5, 0.4, b.box, *f, np.zeros(1))


@pytest.mark.parametrize("graph", [0, 1])
def test_induction_without_polarisable_sites(product, tmp_path, graph):
    b = water_box(Model(data_dir("fs3")), 37, 10.37, 9, ld=28)
    m = _model(tmp_path, charges=True, npol=0)
    with Context(m, b.nm, b.box) as c:
        c.set_option("graph_loop", graph)
        with pytest.raises(CcpError, match="invalid configuration"):
            c.hot_path(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box)
