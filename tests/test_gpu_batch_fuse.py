"""Option fuse_fs3 of a batch: a call with parameter gradients returns them whether or not the
option fs3_param_grad is on, in boxes whose FS3 is fused (by triples) and in wider ones, where FS3
runs per frame by pairs.

The same kernels add the same terms; only the order of atomic additions differs between two runs
(some 1e-14 of a sum's size; 1e-12 of energies and forces and 1e-11 of gradients, whose entries
cancel more, are test_gpu_batch_c4's bounds)."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Batch, Model, _lib, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import water_box

from conftest import rel

pytestmark = pytest.mark.gpu

NF = 3


@pytest.mark.parametrize("nm,L", [(37, 10.37), (128, 15.64)])
def test_gradients_without_the_option(product, nm, L):
    import torch
    m = Model(data_dir("fs3"))
    boxes = [water_box(m, nm, L, 50 + f) for f in range(NF)]
    args = [torch.as_tensor(np.stack([getattr(b, k) for b in boxes]), device="cuda")
            for k in ("x", "y", "z", "xs", "ys", "zs")]
    res = []
    for fuse, option in ((1, 0), (0, 1)):
        f = [torch.zeros_like(args[3]) for _ in range(3)]
        pg = np.zeros((NF, 2 * m.get_int("nclass") + 2 * 3 * 289))
        with Batch(m, nm, L, slots=2) as bt:
            bt.set_option("fuse_fs3", fuse)
            bt.set_option("fs3_param_grad", option)
            for _ in range(2):
                for t in f:
                    t.zero_()
                es = bt.terms_device(_lib.TERM_INDUCTION | _lib.TERM_FS3, [L] * NF, *args, *f,
                                     pgrad=pg)
        res.append((es, np.stack([t.cpu().numpy() for t in f]), pg))
    (e1, f1, g1), (e0, f0, g0) = res
    for a, b in zip(e1, e0):
        assert a["fs3pe"] == pytest.approx(b["fs3pe"], rel=1e-12)
        assert a["indpe"] == pytest.approx(b["indpe"], rel=1e-12)
    assert rel(f1, f0) <= 1e-12
    assert rel(g1, g0) <= 1e-11
    assert (np.abs(g0).max(axis=1) > 0).all()


def test_option_is_as_before_after_the_call(product):
    """The gradients of a fused call in wide boxes do not switch the contexts' option on."""
    import ctypes as C
    import torch
    m = Model(data_dir("fs3"))
    boxes = [water_box(m, 128, 15.64, 50 + f) for f in range(2)]
    args = [torch.as_tensor(np.stack([getattr(b, k) for b in boxes]), device="cuda")
            for k in ("x", "y", "z", "xs", "ys", "zs")]
    pg = np.zeros((2, 2 * m.get_int("nclass") + 2 * 3 * 289))
    with Batch(m, 128, 15.64, slots=2) as bt:
        bt.set_option("fuse_fs3", 1)
        bt.terms_device(_lib.TERM_FS3, [15.64] * 2, *args, pgrad=pg)
        assert np.abs(pg).max() > 0
        for s in range(2):
            h, v = C.c_void_p(), C.c_int(-1)
            assert _lib.lib().ccp_batch_context(bt._h, s, C.byref(h)) == 0
            assert _lib.lib().ccp_context_get_option(h, b"fs3_param_grad", C.byref(v)) == 0
            assert v.value == 0
