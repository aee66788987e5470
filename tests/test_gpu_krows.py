"""The Ewald reciprocal sums by k-vector rows (FP64 tensor cores) against the same sums k-vector
by k-vector (dipole_row_form = 0): energy, virial, forces, static field and induction forces at
every number of n tiles, at the first k_max past the form's range, with different k_max per axis,
and for the form on the fixed scratch.

Both form the same products of the same phase tables and add them in a different order, so a
structure factor differs by about sqrt(n) * 1.1e-16 of the sum of its terms' sizes (n < 1000
sites) and the forces, their sums over k, by about 1e-14 of their norm; 1e-12 leaves room for
the cancellation in them.  The dipoles converge to the same fixed point (as in
test_gpu_dipole_forms)."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Context, Model, data_dir
from ccpol23_plus_2025_mbmd_b200.api import kspace_ewald_fixed
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-12
# one to five n tiles with full and with short last ones, past the form's 19, unequal axes
KMAX = [(1, 1, 1), (3, 3, 3), (4, 4, 4), (7, 7, 7), (8, 8, 8), (13, 13, 13), (19, 19, 19),
        (20, 20, 20), (5, 9, 6), (9, 4, 11)]


@pytest.fixture(scope="module")
def box(product):
    m = Model(data_dir("fs3"))
    return m, water_box(m, 37, 10.37, 9, ld=28)


def _kspace(m, b, k, rows):
    f = [np.zeros_like(b.xs) for _ in range(3)]
    vir = np.zeros(1)
    with Context(m, b.nm, b.box, precision="fp64") as c:
        c.set_option("dipole_row_form", rows)
        e = c.kspace_ewald(b.x, b.y, b.z, b.xs, b.ys, b.zs, *k, 0.4, b.box, *f, vir)
    return e, vir[0], np.stack(f)


@pytest.mark.parametrize("k", KMAX)
def test_kspace_ewald(box, k):
    m, b = box
    e, vir, F = _kspace(m, b, k, 1)
    e0, vir0, F0 = _kspace(m, b, k, 0)
    assert abs(e - e0) <= TOL * abs(e0)
    assert abs(vir - vir0) <= TOL * max(abs(vir0), abs(e0))
    assert rel(F, F0) <= TOL


@pytest.mark.parametrize("k", KMAX)
def test_kspace_ewald_fixed(box, k):
    torch = pytest.importorskip("torch")
    m, b = box
    ns = m.ns
    dev = [torch.tensor(np.ascontiguousarray(a), device="cuda")
           for a in (b.x, b.y, b.z, b.xs[:, :ns], b.ys[:, :ns], b.zs[:, :ns])]
    f = [torch.zeros((b.nm, ns), dtype=torch.float64, device="cuda") for _ in range(3)]
    q, vir = (torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(2))
    kspace_ewald_fixed(m, *dev, *k, 0.4, b.box, q, *f, vir,
                       torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    e0, vir0, F0 = _kspace(m, b, k, 0)
    assert abs(q.item() - e0) <= TOL * abs(e0)
    assert abs(vir.item() - vir0) <= TOL * max(abs(vir0), abs(e0))
    assert rel(torch.stack(f).cpu().numpy(), F0[:, :, :ns]) <= TOL


@pytest.mark.parametrize("k", KMAX)
@pytest.mark.parametrize("nm,L", [(37, 10.37), (200, 18.15)])
def test_induction(product, nm, L, k):
    m = Model(data_dir("fs3"))
    b = water_box(m, nm, L, 400 + nm, ld=28)
    res = []
    for rows in (1, 0):
        out = [np.zeros_like(b.xs) for _ in range(6)]
        vir = np.zeros(1)
        with Context(m, nm, b.box, precision="fp64") as c:
            c.set_option("dipole_row_form", rows)
            c.set_ewald(0.35, *k)
            e, it = c.nb_induction(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box, *out, vir)
        res.append((e, it, np.stack(out[:3]), np.stack(out[3:]), vir[0]))
    (e, it, mu, F, vir), (e0, it0, mu0, F0, vir0) = res
    assert it == it0
    assert abs(e - e0) <= TOL * abs(e0)
    assert rel(mu, mu0) <= TOL
    assert rel(F, F0) <= TOL
    assert abs(vir - vir0) <= TOL * max(abs(vir0), abs(e0))
