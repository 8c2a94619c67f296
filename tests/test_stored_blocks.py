"""Stored blocks (k_blk1, the 64-wide passes, the panels between) against the same product in
64-bit torch from the same representation (perf/cases.py): images with fewer blocks than CTA
slots (tasks of 64-row chunks) and with more, blocks of odd sizes below and above one tile
of 64 and one unit of 128, level-mismatched pairs, every panel width and remainder.

Tolerance: FP64 as the on-the-fly path's (1e-13); mixed 2e-6 (FP32 blocks, BF16x3 or 3xTF32
products with FP32 sums of at most 64 terms).
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,n,leaf", [("coulomb", 20, 100), ("coulomb", 1501, 300), ("coulomb", 2003, 40),
                                           ("gaussian", 5000, 700), ("matern32", 12007, 150), ("rpy", 130, 50),
                                           ("rpy", 3001, 60)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_matches_64_bit_product(kernel, n, leaf, precision):
    import torch
    from perf import cases
    case = {"kind": "apply", "kernel": kernel, "n": n, "leaf": leaf, "mode": "generate", "precision": precision, "api": "device"}
    rep = cases.Rep(case, n, 4)
    img = cases.Image(rep.describe(), precision, blocks="generate")
    X = cases._rhs(case, rep.kd * n, 128, 4)
    Y = rep.apply(X)
    tol = 1e-13 if precision == "fp64" else 2e-6
    for nv in (1, 2, 3, 4, 8, 16, 20, 33, 64, 100):
        y = img.matmul_device(X[:, :nv].contiguous())
        torch.cuda.synchronize()
        assert float((y - Y[:, :nv]).norm() / Y[:, :nv].norm()) < tol, nv
    # host calls: through the pinned buffer and past its size, both layouts
    import numpy as np
    Xh, Yh = X.cpu().numpy(), Y.cpu().numpy()
    assert np.linalg.norm(img.matvec(Xh[:, 0]) - Yh[:, 0]) < tol * np.linalg.norm(Yh[:, 0])
    for layout in (101, 102):
        for nv in (2, 17):
            assert np.linalg.norm(img.matmul(Xh[:, :nv], layout) - Yh[:, :nv]) < tol * np.linalg.norm(Yh[:, :nv])
    img.close()


def test_few_large_blocks_fit_the_no_allocation_apply():
    """36 near blocks of 3,000 columns: tasks small enough to fill the GPU would have 2.6 million
    slots, past that apply's work space; such an image keeps its tall tasks (same sums in another
    order, 1e-13)."""
    import torch
    from perf import cases
    case = {"kind": "apply", "kernel": "coulomb", "n": 24000, "leaf": 8000, "mode": "generate", "precision": "fp64", "api": "device"}
    rep = cases.Rep(case, 24000, 4)
    img = cases.Image(rep.describe(), "fp64", blocks="generate")
    x = cases._rhs(case, 24000, 1, 4)[:, 0].contiguous()
    y0, y = img.matmul_device(x[:, None].contiguous())[:, 0], torch.empty_like(x)
    img.matvec_device_noalloc(x, y)
    torch.cuda.synchronize()
    assert float((y - y0).norm() / y0.norm()) < 1e-13
    img.close()


@pytest.mark.parametrize("kernel,n,leaf,mode", [("coulomb", 6000, 300, "given"), ("coulomb", 6000, 300, "generate"),
                                                ("gaussian", 20000, 400, "jit")])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_an_apply_right_after_create_sees_whole_uploads(kernel, n, leaf, mode, precision):
    """The caller's arrays are overwritten as soon as create returns, and the first apply starts at
    once on the image's own stream."""
    import numpy as np
    import torch
    from perf import cases
    case = {"kind": "apply", "kernel": kernel, "n": n, "leaf": leaf, "mode": mode, "precision": precision, "api": "host"}
    rep = cases.Rep(case, n, 6)
    X = cases._rhs(case, n, 8, 6)
    Y, Xh = rep.apply(X).cpu().numpy(), X.cpu().numpy()
    d = rep.describe(mode == "given")
    torch.cuda.synchronize()
    img = cases.Image(d, precision, blocks="generate" if mode == "generate" else "given")
    for a in rep.host.values():
        a.fill(np.nan if a.dtype == np.float64 else 0)
    assert np.linalg.norm(img.matmul(Xh) - Y) < (1e-13 if precision == "fp64" else 2e-6) * np.linalg.norm(Y)
    img.close()


def test_lists_of_warp_and_cta_tasks():
    """Near blocks of about 181 x 181 FP32 values, on both sides of one warp's 128 KB (blk1_fits): a
    list with tasks of both kinds, whose two launches cover it (2e-6 as above)."""
    import numpy as np
    import torch
    from perf import cases
    n = 92672
    case = {"kind": "apply", "kernel": "coulomb", "n": n, "leaf": 300, "mode": "generate", "precision": "mixed", "api": "device"}
    rep = cases.Rep(case, n, 5)
    npt = (rep.t["end"] - rep.t["start"])[rep.t["n_child"] == 0]
    assert 4 * int(npt.min()) ** 2 <= 128 * 1024 < 4 * int(npt.max()) ** 2
    img = cases.Image(rep.describe(), "mixed", blocks="generate")
    x = cases._rhs(case, n, 1, 5)
    y, e = img.matmul_device(x), rep.apply(x)
    torch.cuda.synchronize()
    assert float((y - e).norm() / e.norm()) < 2e-6
    assert np.linalg.norm(img.matvec(x[:, 0].cpu().numpy()) - e[:, 0].cpu().numpy()) < 2e-6 * float(e.norm())
    img.close()


@pytest.mark.parametrize("kernel,n,mode,precision,variant", [
    ("coulomb", 6000, "generate", "fp64", None), ("coulomb", 6000, "generate", "mixed", None), ("coulomb", 200, "generate", "mixed", None),
    ("gaussian", 20000, "jit", "fp64", None), ("gaussian", 20000, "jit", "mixed", "tc"), ("gaussian", 20000, "jit", "mixed", "pair")])
def test_phase_times_add_up(kernel, n, mode, precision, variant):
    """h2gpu_get_stats: the phases of any number of applies add up to their device time, with the
    near field beside the others, one after the other (pair), and without admissible pairs."""
    from perf import cases
    case = {"kind": "apply", "kernel": kernel, "n": n, "leaf": 300, "mode": mode, "precision": precision, "api": "device"}
    rep = cases.Rep(case, n, 4)
    img = cases.Image(rep.describe(), precision, blocks="generate" if mode == "generate" else "given")
    if variant:
        img.set_jit_variant(variant)
    for nv in (1, 16, 64):
        X = cases._rhs(case, n, nv, 4)
        img.matmul_device(X)
        img.reset_stats()
        for _ in range(3):
            img.matmul_device(X)
        st = img.stats()
        assert st["ms_total"] > 0 and min(st["ms_phase"]) >= 0
        assert abs(sum(st["ms_phase"]) - st["ms_total"]) < 1e-4 * st["ms_total"], (nv, st["ms_phase"], st["ms_total"])
    img.close()
