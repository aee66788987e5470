"""FS3's pair form in contexts whose lists overflow and grow, against FS3 by triples in a context
of its own: energy, counts, site and COM forces, virial.

The two add the same terms in different orders; 1e-10 is the bound that test_gpu_fs3_pairs derives
for them."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import CcpError, Context, Model, _lib, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _fs3(c, b):
    import torch
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    f = [torch.zeros(b.xs.shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    c3 = [torch.zeros(b.nm, dtype=torch.float64, device="cuda") for _ in range(3)]
    e = c.terms_device(_lib.TERM_FS3, *(T(getattr(b, k)) for k in ("x", "y", "z", "xs", "ys", "zs")),
                       b.box, *f, None, None, None, *c3)
    return e, np.stack([t.cpu().numpy() for t in f]), np.stack([t.cpu().numpy() for t in c3])


def _compare(r, r0):
    (e, f, c3), (e0, f0, c0) = r, r0
    assert e["n_fs3_triples"] == e0["n_fs3_triples"] > 0
    assert e["n_fs3_blend"] == e0["n_fs3_blend"]
    assert abs(e["fs3pe"] - e0["fs3pe"]) <= TOL * abs(e0["fs3pe"])
    assert abs(e["vir"] - e0["vir"]) <= TOL * abs(e0["vir"])
    assert rel(f, f0) <= TOL
    assert rel(c3, c0) <= TOL


def _triples(m, b):
    with Context(m, b.nm, b.box) as c:
        c.set_option("fs3_pair_form", 0)
        return _fs3(c, b)


def _with_rcut(tmp_path, rcut):
    """The FS3 model with another cut-off radius in its CONTROL."""
    for p in data_dir("fs3").iterdir():
        t = p.read_text()
        if p.name == "CONTROL":
            assert t.count("9.0                 # rcut ") == 1
            t = t.replace("9.0                 # rcut ", f"{rcut:.1f}                # rcut ")
        (tmp_path / p.name).write_text(t)
    return Model(tmp_path)


def test_neighbour_list_overflow(product, tmp_path):
    """A neighbour list that outgrows its first 192 entries per molecule lacks pairs of triples
    that it holds; the evaluation that follows with a longer list still goes by pairs."""
    m = _with_rcut(tmp_path, 12.0)
    b = water_box(m, 300, 20.79, 702, ld=28)  # 244 neighbours per molecule
    ref = _triples(m, b)
    with Context(m, b.nm, b.box) as c:
        _compare(_fs3(c, b), ref)
        assert c.get_option("fs3_pair_form_active") == 1


@pytest.mark.parametrize("grad", [0, 1])
@pytest.mark.parametrize("before", [None, 0, 1])
def test_pair_list_overflow(product, before, grad):
    """A box of some 26 pairs per molecule, more than the pair list holds at first, in a new
    context and in one whose triple records hold those of an earlier box, by triples (0) or by
    pairs (1): the records that the overflowing evaluation does not fill are not read."""
    m = Model(data_dir("fs3"))
    dense = water_box(m, 100, 12.65, 700, ld=28, min_oo=2.2)
    ref = _triples(m, dense)
    with Context(m, 100, 14.41) as c:
        if before is not None:
            c.set_option("fs3_pair_form", before)
            b = water_box(m, 100, 14.41, 701, ld=28)
            _compare(_fs3(c, b), _triples(m, b))
        c.set_option("fs3_pair_form", 1)
        c.set_option("fs3_param_grad", grad)
        for _ in range(2):
            _compare(_fs3(c, dense), ref)
            assert c.get_option("fs3_pair_form_active") == 1


def test_memory_bound(product):
    """Pair tables above the bound of option fs3_pair_mib: FS3 runs by triples, also where they
    outgrow it only once a dense box's pairs are known (57 MiB for the first 2000 pairs of 100
    molecules, some 85 for the 26 each that it has)."""
    m = Model(data_dir("fs3"))
    dense = water_box(m, 100, 12.65, 700, ld=28, min_oo=2.2)
    ref = _triples(m, dense)
    with Context(m, 100, dense.box) as c:
        with pytest.raises(CcpError, match="negative"):
            c.set_option("fs3_pair_mib", -1)
        for mib, active in ((32, 0), (64, 0), (0, 1), (256, 1), (32, 0), (256, 1)):
            c.set_option("fs3_pair_mib", mib)
            assert c.get_option("fs3_pair_mib") == mib
            for _ in range(2):
                _compare(_fs3(c, dense), ref)
                assert c.get_option("fs3_pair_form_active") == active
