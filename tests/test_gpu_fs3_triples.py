"""FS3 by triples in boxes where the pair form is the default (option fs3_pair_form = 0): blocks of
several triples against blocks of one, the FP32 gradient passes of the mixed form against FP64, and
a batch with FS3 fused over its frames against single frames.

Runs of the same kernel differ in the order of their atomic additions only (1e-12, gradients 1e-11,
as in test_gpu_streams and test_gpu_batch_c4).  The FP32 passes leave the energy and the COM forces
alone; they round products of site forces to 2^-24, which shows above 1e-9 of the force norm, and
the site forces stay within the mixed form's 1e-5, as in test_gpu_mixed."""
import numpy as np
import pytest

from ccpol23_plus_2025_mbmd_b200 import Batch, Context, Model, _lib, data_dir
from ccpol23_plus_2025_mbmd_b200.generator import CONFIGS, water_box

from conftest import rel

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _fs3(m, b, precision, **opts):
    import torch
    args = [_dev(getattr(b, k)) for k in ("x", "y", "z", "xs", "ys", "zs")]
    f = [torch.zeros_like(args[3]) for _ in range(3)]
    c3 = [torch.zeros_like(args[0]) for _ in range(3)]
    with Context(m, b.nm, b.box, precision=precision) as c:
        c.set_option("fs3_pair_form", 0)
        for k, v in opts.items():
            c.set_option(k, v)
        e = c.terms_device(_lib.TERM_FS3, *args, b.box, *f, None, None, None, *c3)
        assert c.get_option("fs3_pair_form_active") == 0
    return e, np.stack([t.cpu().numpy() for t in f]), np.stack([t.cpu().numpy() for t in c3])


@pytest.mark.parametrize("precision,fp32_passes", [("fp64", 0), ("mixed", 0), ("mixed", 1)])
def test_table_reuse_matches_single_triple_blocks(product, precision, fp32_passes):
    m = Model(data_dir("fs2fs3"))
    b = water_box(m, 128, 15.64, 77, ld=28)
    (e8, f8, c8), (e1, f1, c1) = (_fs3(m, b, precision, fs3_triples_per_block=t,
                                       fs3_fp32_passes=fp32_passes) for t in (8, 1))
    assert e8["fs3pe"] == pytest.approx(e1["fs3pe"], rel=1e-12)
    assert e8["vir"] == pytest.approx(e1["vir"], rel=1e-12)
    assert rel(f8, f1) <= 1e-12
    assert rel(c8, c1) <= 1e-12


def test_fp32_passes_against_fp64(product):
    cfg = CONFIGS["c2_512"]
    m = Model(data_dir(cfg["variant"]))
    b = water_box(m, cfg["nm"], cfg["box"], cfg["seed"])
    (e0, f0, c0), (e1, f1, c1) = (_fs3(m, b, "mixed", fs3_fp32_passes=p) for p in (0, 1))
    assert e1["fs3pe"] == pytest.approx(e0["fs3pe"], rel=1e-12)
    assert rel(c1, c0) <= 1e-12
    assert 1e-9 < rel(f1, f0) <= 1e-5


def test_fp32_passes_at_2048(product):
    """The per-molecule forces with the FP32 passes, 1.45e-5 off at 2048 waters, where the mixed
    form's bar is 1e-5: the reason why they are not its default."""
    cfg = CONFIGS["c5_2048"]
    m = Model(data_dir(cfg["variant"]))
    b = water_box(m, cfg["nm"], cfg["box"], cfg["seed"])
    F = []
    for precision, opt in (("fp64", 0), ("mixed", 1)):
        with Context(m, b.nm, b.box, precision=precision) as c:
            c.set_option("fs3_pair_form", 0)
            c.set_option("fs3_fp32_passes", opt)
            r = c.hot_path(b.x, b.y, b.z, b.xs, b.ys, b.zs, b.box)
            assert c.get_option("fs3_pair_form_active") == 0
        f = np.stack([r.fxs, r.fys, r.fzs])
        F.append((f, f.sum(2) + np.stack([r.fxfs2, r.fyfs2, r.fzfs2]) +
                  np.stack([r.fxfs3, r.fyfs3, r.fzfs3])))
    (f0, t0), (f1, t1) = F
    assert rel(f1, f0) <= 1e-5
    assert 1e-9 < rel(t1, t0) <= 2e-5


def test_fused_batch_equals_single_frames(product):
    """Frames of 256 waters, three-body and induction terms with parameter gradients: FS3 of all
    frames in one launch (its own neighbour lists, triples and sums per frame)."""
    import torch
    nf, cfg = 8, CONFIGS["c4_256"]
    m = Model(data_dir(cfg["variant"]))
    boxes = [water_box(m, cfg["nm"], cfg["box"], cfg["seed"] + f) for f in range(nf)]
    args = [_dev(np.stack([getattr(b, k) for b in boxes])) for k in ("x", "y", "z", "xs", "ys", "zs")]
    terms = _lib.TERM_INDUCTION | _lib.TERM_FS3 | _lib.TERM_FS2
    ncoef = m.get_int("nclass")

    def outputs(a):
        return ([torch.zeros_like(a[3]) for _ in range(3)] + [torch.zeros_like(a[0]) for _ in range(6)] +
                [torch.zeros_like(a[3]) for _ in range(3)])

    out = outputs(args)
    pg = np.zeros((nf, 2 * ncoef + 2 * 3 * 289))
    with Batch(m, cfg["nm"], cfg["box"], slots=4) as bt:
        bt.set_option("fs3_pair_form", 0)
        bt.set_option("fuse_fs3", 1)
        es = bt.terms_device(terms, [cfg["box"]] * nf, *args, *out, pgrad=pg)
    got = [t.cpu().numpy() for t in out]
    with Context(m, cfg["nm"], cfg["box"]) as c:
        c.set_option("fs3_pair_form", 0)
        c.set_option("fs3_param_grad", 1)
        for f in range(nf):
            a1 = [a[f].contiguous() for a in args]
            o1 = outputs(a1)
            e1 = c.terms_device(terms, *a1, cfg["box"], *o1)
            for k in ("indpe", "fs2pe", "fs3pe", "vir"):
                assert es[f][k] == pytest.approx(e1[k], rel=1e-12, abs=1e-12), (f, k)
            for k in ("ind_iters", "n_fs3_triples", "n_fs3_blend"):
                assert es[f][k] == e1[k], (f, k)
            for g, a in zip(got, o1):
                assert rel(g[f], a.cpu().numpy()) <= 1e-12, f
            assert rel(pg[f], np.concatenate([np.ravel(p) for p in c.fs3_param_grad()])) <= 1e-11
