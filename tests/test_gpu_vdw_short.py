"""The 2-body term where its short-range damping is at work on all, some and none of the site
pairs: two molecules at falling distances against the oracle.  The tolerance is the parity
tests' (1e-10): the terms' exponents reach 30, so that a distance's rounding grows to some 1e-14
of a term, and the terms of both signs cancel to a few per cent of their size."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.mark.parametrize("d", [0.9, 1.4, 1.9, 2.4, 2.9, 3.6, 6.0])
def test_two_molecules(product, oracle, d):
    O = oracle
    m = Model(data_dir("fs3"))
    L = 20.0
    b = water_box(m, 2, L, 5, ld=28)
    b.x[:], b.y[:], b.z[:] = [0.0, d * 0.6], [0.0, -d * 0.48], [0.0, d * 0.64]
    M = O.make_model(O.read_inputs(data_dir("fs3")), 2, L)
    st = O.State(2, b.xs.shape[1])
    eo = O.ccpol23plus(M, b.x, b.y, b.z, b.xs, b.ys, b.zs, L, st)
    f = [np.zeros_like(b.xs) for _ in range(3)]
    vir = np.zeros(1)
    with Context(m, 2, L, precision="fp64") as c:
        e = c.ccpol23plus(b.x, b.y, b.z, b.xs, b.ys, b.zs, L, *f, vir)
    assert abs(e - eo) <= TOL * abs(eo)
    assert rel(np.stack(f), np.stack([st.fxs, st.fys, st.fzs])) <= TOL
    assert abs(vir[0] - st.vir.value) <= TOL * abs(st.vir.value)
