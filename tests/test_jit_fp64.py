"""The FP64 on-the-fly kernels (k_jit64) against the same product in 64-bit torch from the same
representation (perf/cases.py): every panel width and remainder, target chunks of few and
of 128 points (leaves of 100 and 400), images with fewer chunks than the GPU has CTA slots
(clusters share a chunk), and kernel arguments outside the fast evaluation's range (r = 0;
exponents below -700).

Tolerance: sums of at most 27 x 400 + 189 x 400 terms of both signs, each kernel value within
a few units of 1.1e-16 (relative to its largest exponent, below 700), and a transfer matrix
product per level: 1e-13 covers 1e3 units; the drop-in's bar is 1e-12.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,param", [("coulomb", 1.0), ("gaussian", 1.0), ("gaussian", 8.0), ("matern32", 1.0),
                                          ("matern32", 40.0), ("rpy", 1.0)])
@pytest.mark.parametrize("n,leaf", [(33, 100), (129, 400), (1500, 100), (6001, 400), (20000, 100)])
def test_matches_64_bit_product(kernel, param, n, leaf):
    import torch
    from perf import cases
    case = {"kind": "apply", "kernel": kernel, "n": n, "leaf": leaf, "mode": "jit", "precision": "fp64", "param": param,
            "api": "device"}
    rep = cases.Rep(case, n, 2)
    img = cases.Image(rep.describe(), "fp64")
    X = cases._rhs(case, rep.kd * n, 21, 2)
    Y = rep.apply(X)
    for nv in (1, 2, 3, 4, 7, 8, 16, 21):
        y = img.matmul_device(X[:, :nv].contiguous())
        torch.cuda.synchronize()
        assert float((y - Y[:, :nv]).norm() / Y[:, :nv].norm()) < 1e-13, nv
    img.close()


@pytest.mark.parametrize("kernel", ["coulomb", "gaussian", "matern32", "rpy"])
@pytest.mark.parametrize("n,leaf", [(40, 100), (1500, 300), (9000, 100)])
def test_mixed_small_images(kernel, n, leaf):
    """FP32 evaluation with clusters of 2 to 8 CTAs per chunk, every panel width, on the CUDA
    and the tensor cores: the mixed path's 2e-6 (FP32 kernel values, 3xTF32 products)."""
    import torch
    from perf import cases
    case = {"kind": "apply", "kernel": kernel, "n": n, "leaf": leaf, "mode": "jit", "precision": "mixed", "api": "device"}
    rep = cases.Rep(case, n, 3)
    img = cases.Image(rep.describe(), "mixed")
    X = cases._rhs(case, rep.kd * n, 16, 3)
    Y = rep.apply(X)
    for variant in ("tc", "simt"):
        img.set_jit_variant(variant)
        for nv in (1, 2, 4, 5, 8, 16):
            y = img.matmul_device(X[:, :nv].contiguous())
            torch.cuda.synchronize()
            assert float((y - Y[:, :nv]).norm() / Y[:, :nv].norm()) < 2e-6, (variant, nv)
    img.close()
