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


def _entries(kernel, P, param=1.0):
    """K of the points P (n, 3) as the engine evaluates it: the image of one leaf, applied to unit
    vectors (each sum has one term that is not zero, so an entry is the kernel's value)."""
    import numpy as np
    import torch
    from perf import cases
    n = len(P)
    case = {"kind": "apply", "kernel": kernel, "n": n, "leaf": n, "mode": "jit", "precision": "fp64", "param": param,
            "api": "device"}
    rep = cases.Rep(case, n, 1)
    rep.points = np.ascontiguousarray(P[rep.t["order"]])       # P in the caller's order
    img = cases.Image(rep.describe(), "fp64")
    E = torch.eye(img.N, dtype=torch.float64, device="cuda")
    K = img.matmul_device(E)
    if kernel != "rpy":                                        # the matrix path and the multiply-add's
        assert torch.equal(K[:, :1], img.matmul_device(E[:, :1].contiguous()))
    torch.cuda.synchronize()
    img.close()
    return K.cpu().numpy()


def _on_a_line(x):
    import numpy as np
    P = np.zeros((len(x), 3))
    P[:, 0] = x
    d = x[:, None] - x[None, :]
    return P, d * d                                            # r^2 exactly as the kernel rounds it


def _ulps(v, exact):
    """Largest distance of v from exact (extended precision) in units of exact's last place in FP64
    (of the smallest normal number's below it)."""
    import numpy as np
    u = np.maximum(np.spacing(np.abs(exact).astype(np.float64)), np.spacing(0.0)).astype(np.longdouble)
    return float((np.abs(v.astype(np.longdouble) - exact) / u).max())


def test_fp64_kernel_values_entry_by_entry():
    """Every value, not a norm: the FP64 exponential, reciprocal square root and square root of the
    kernels over their whole ranges and on both sides of each range's end (exponents of -700,
    below which results are subnormal and then zero; zero and subnormal r^2), against extended precision.

    Bounds in units of the last place: Gaussian (its exponent -r^2 is exact for l = 1) 1.25, where
    CUDA's exp documents 1 (the 16-entry table's value, its polynomial and one rounding
    come to 1.09); Coulomb 1, as CUDA's rsqrt.  Matern, relative, in 2^-52: the exponent carries
    half from the square root and half from its product, which the exponential turns into
    |t|, and three more come from the exponential, 1 - t and their product; where e^t is
    subnormal (|t| > 708) its last unit times 1 - t and the product's rounding are another
    2 + |t| times 2^-1074."""
    import numpy as np
    import torch
    rng = np.random.default_rng(3)
    ld = np.longdouble

    # exp: r^2 from 1e-18 to 760, dense around 700
    x = np.concatenate([[0.0], 10.0 ** rng.uniform(-9, 1.4, 300), rng.uniform(20, 27.6, 150), np.sqrt(700 + rng.uniform(-1, 1, 61))])
    P, r2 = _on_a_line(x)
    K, e = _entries("gaussian", P), np.exp(-r2.astype(ld))
    assert _ulps(K, e) < 1.25
    cuda = torch.exp(-torch.from_numpy(r2).cuda()).cpu().numpy()
    assert _ulps(K, e) < _ulps(cuda, e) + 0.5
    # exponents above zero as well (l < 0): up to e^700
    K, e = _entries("gaussian", P[:300], -1.0), np.exp(r2[:300, :300].astype(ld))
    assert _ulps(K, e) < 1.25

    # rsqrt: r from 1e-162 (r^2 subnormal; zero below) to 1e150, coincident points 0
    x = np.concatenate([[0.0, 0.0], 10.0 ** rng.uniform(-162, -150, 60), 10.0 ** rng.uniform(-150, 150, 300), 10.0 ** rng.uniform(-3, 3, 150)])
    P, r2 = _on_a_line(x)
    K = _entries("coulomb", P)
    normal = r2 >= 2.0 ** -1022
    assert (K[r2 == 0] == 0).all()
    assert _ulps(K[normal], 1 / np.sqrt(r2[normal].astype(ld))) < 1.0
    low = (r2 > 0) & ~normal
    assert low.any() and _ulps(K[low], 1 / np.sqrt(r2[low].astype(ld))) < 2.0

    # sqrt and exp together, past |t| = 700 (r = 404)
    x = np.concatenate([[0.0], 10.0 ** rng.uniform(-160, -3, 40), 10.0 ** rng.uniform(-3, 2.6, 300), rng.uniform(380, 440, 171)])
    P, r2 = _on_a_line(x)
    K = _entries("matern32", P)
    t = ld(-1.7320508075688772) * np.sqrt(r2.astype(ld))
    e = (1 - t) * np.exp(t)
    bound = (3 + np.abs(t)) * ld(2) ** -52 * e + np.where(t < -708, 2 + np.abs(t), 1) * ld(2) ** -1074
    assert float((np.abs(K - e) / bound).max()) < 1.0

    # RPY: spheres apart, touching and overlapping, any direction; a block's entries relative to
    # its largest, 16 units (r^2 of three products, 1 / r, the two coefficients, three products)
    n = 120
    P = rng.standard_normal((n, 3))
    P *= (10.0 ** rng.uniform(-2, 3, n) / np.linalg.norm(P, axis=1))[:, None]
    P[1::3] = P[::3][:40] + 2.0 * (1 + 1e-9 * rng.uniform(-1, 1, 40))[:, None] * np.eye(3)[rng.integers(0, 3, 40)]
    K = _entries("rpy", P).reshape(n, 3, n, 3).transpose(0, 2, 1, 3).astype(ld)
    d = (P[:, None] - P[None]).astype(ld)
    r = np.sqrt((d * d).sum(-1))
    i = np.where(r > 0, 1 / np.where(r > 0, r, 1), 0)
    c = 1 / ld(6 * np.pi * (1.0 / (6.0 * np.pi)))
    far = r > 2
    t1 = np.where(far, c * ld(0.75) * i * (1 + 2 * i * i / 3), c * (1 - 9 * r / 32))
    t2 = np.where(far, c * ld(0.75) * i * (1 - 2 * i * i), c * 3 * r / 32)
    h = d * i[..., None]
    E = t2[..., None, None] * h[..., :, None] * h[..., None, :] + t1[..., None, None] * np.eye(3)
    assert float((np.abs(K - E).max((-1, -2)) / np.abs(E).max((-1, -2))).max()) < 16 * 2.0 ** -52
