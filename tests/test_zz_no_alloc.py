"""The no-allocation apply (h2gpu_matvec_device_noalloc) against the regular device
apply (h2gpu_matmul_device) of the same image.

The no-allocation entry point is for callers that cannot allocate device memory when
they apply the matrix (device memory owned by another allocator, or code that must not
stall on cudaMalloc/cudaFree, which synchronize the device).  Its work buffers live in a
fixed 16 MiB device array of the library; it must give the same result as the regular
path on two calls in a row (the array keeps the previous call's contents), and reject
images that need more work space.  This file is collected last on purpose.
"""
import os

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def image_from(name, precision="fp64"):
    from oracle import oracle as O
    from h2pack_b200 import Image
    z = np.load(os.path.join(GOLDEN, name + ".npz"))
    keep = ("x", "y_ref", "X", "Y_ref", "coord_in", "reltol")
    h = O.DescHolder({k: (int(z[k]) if z[k].ndim == 0 else z[k]) for k in z.files if k not in keep})
    return Image(h.desc, precision=precision), h


@pytest.mark.parametrize("name,precision", [("coulomb_aot", "fp64"), ("matern32_jit", "fp64"),
                                            ("rpy_jit", "fp64"), ("gaussian_jit", "mixed")])
def test_noalloc_matches_regular_apply_twice(name, precision):
    import torch
    img, _h = image_from(name, precision)
    try:
        g = torch.Generator(device="cuda").manual_seed(5)
        x = torch.randn(img.N, 1, dtype=torch.float64, device="cuda", generator=g)
        y_ref = img.matmul_device(x)            # regular path (allocates its work buffers)
        torch.cuda.synchronize()
        y_ref = y_ref[:, 0].cpu().numpy()
        x0 = x[:, 0].contiguous()
        ys = [torch.full((img.N,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(3)]
        torch.cuda.synchronize()
        free_before = None
        for y in ys:                            # the scratch keeps the previous call's contents
            img.matvec_device_noalloc(x0, y)
            torch.cuda.synchronize()
            if free_before is None:
                # the first call on the device may load the library's device module (and
                # with it the scratch array); later calls allocate nothing on the device
                free_before = torch.cuda.mem_get_info()[0]
            else:
                assert torch.cuda.mem_get_info()[0] == free_before
            assert rel(y.cpu().numpy(), y_ref) < 1e-12
    finally:
        img.close()


def test_noalloc_rejects_images_beyond_the_limit():
    import torch
    from conftest import make_points
    from h2pack_b200 import H2Matrix
    H = H2Matrix("coulomb", make_points("coulomb", 40000, 3), [], 1e-6, BD_JIT=0, max_leaf_points=300)
    try:
        img = H.image()
        x = torch.zeros(H.N, dtype=torch.float64, device="cuda")
        y = torch.zeros_like(x)
        with pytest.raises(RuntimeError, match="limited to"):
            img.matvec_device_noalloc(x, y)
    finally:
        H.close()


def test_noalloc_refuses_mixed_image_before_its_first_apply():
    """A mixed-precision image holds FP32 copies of U/B/D only after one allocating
    apply; before that the no-allocation entry point refuses it (status STATE) and
    leaves the caller's current device unchanged."""
    import torch
    img, _h = image_from("coulomb_aot", "mixed")
    try:
        x = torch.randn(img.N, dtype=torch.float64, device="cuda")
        y = torch.zeros_like(x)
        dev = torch.cuda.current_device()
        with pytest.raises(RuntimeError, match="STATE"):
            img.matvec_device_noalloc(x, y)
        assert torch.cuda.current_device() == dev
        img.matmul_device(x[:, None].contiguous())     # makes the FP32 copies
        img.matvec_device_noalloc(x, y)
        torch.cuda.synchronize()
        assert torch.isfinite(y).all()
    finally:
        img.close()


class Captures:
    """Relaxed captures of torch streams, all ended when the block is left, then replayed."""

    def __enter__(self):
        from cuda.bindings import runtime as rt
        self.rt, self.open, self.graphs = rt, [], []
        return self

    def _do(self, r):
        assert r[0] == self.rt.cudaError_t.cudaSuccess, r[0]
        return r[-1]

    def begin(self):
        import torch
        s = torch.cuda.Stream()
        self._do(self.rt.cudaStreamBeginCapture(s.cuda_stream, self.rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed))
        self.open.append(s)
        return s

    def __exit__(self, *err):
        ends = [self.rt.cudaStreamEndCapture(s.cuda_stream) for s in self.open]
        if err[0] is None:
            self.graphs = [self._do(r) for r in ends]

    def replay(self):
        for g, s in zip(self.graphs, self.open):
            ex = self._do(self.rt.cudaGraphInstantiate(g, 0))
            self._do(self.rt.cudaGraphLaunch(ex, s.cuda_stream))
            s.synchronize()
            self._do(self.rt.cudaGraphExecDestroy(ex))
            self._do(self.rt.cudaGraphDestroy(g))


@pytest.mark.parametrize("kernel,mode,precision", [("coulomb", "jit", "fp64"), ("gaussian", "jit", "mixed"),
                                                   ("coulomb", "generate", "fp64"), ("coulomb", "generate", "mixed")])
def test_an_open_capture_leaves_the_image_free(kernel, mode, precision):
    """The no-allocation apply captured on a caller's stream: until that capture ends, the image
    takes applies on other streams, host calls and a second capture, and both graphs replay to
    the eager result."""
    import torch
    from perf import cases
    case = {"kind": "apply", "kernel": kernel, "n": 6000, "leaf": 300, "mode": mode, "precision": precision, "api": "device"}
    rep = cases.Rep(case, 6000, 9)
    assert len(rep.adm)
    img = cases.Image(rep.describe(), precision, blocks="generate" if mode == "generate" else "given")
    X = cases._rhs(case, 6000, 2, 9)
    Y, x = img.matmul_device(X), X[:, 0].contiguous()
    y0 = img.matmul_device(x[:, None])[:, 0].clone()
    Y2, y1, y2, y3 = torch.empty_like(Y), torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    img.matvec_device_noalloc(x, y3)
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    xh = x.cpu().numpy()
    with Captures() as c:
        img.matvec_device_noalloc(x, y1, stream=c.begin())
        img.matmul_device(X, Y2, stream=other)
        img.matvec_device_noalloc(x, y2, stream=c.begin())
        yh = img.matvec(xh)
    torch.cuda.synchronize()
    c.replay()
    same = 1e-13 if precision == "fp64" else 2e-6
    assert rel(Y2.cpu(), Y.cpu()) < same and rel(yh, y0.cpu()) < same
    for y in (y1, y2, y3):
        assert rel(y.cpu(), y0.cpu()) < same
    img.close()
