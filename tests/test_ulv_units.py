"""The ULV solve's units of 64 rows (h2gpu_ulv.cu) at their edges: single nodes just below, at
and above one and two blocks, trees whose nodes have odd sizes, short last blocks and
eliminated parts of any size, every op, Cholesky and LU, against the same solve in 64-bit
torch (perf/cases.py: the factors, and Q applied from its reflectors by torch).

Tolerance: a solve is two sweeps of at most 3 levels, each a product and a substitution of
length m <= 700 with condition below 10: 6 x 700 x 1.1e-16 x 10 < 5e-12 in the worst case,
growing as the square root of the length in practice: 1e-13.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lu", [False, True])
@pytest.mark.parametrize("n,leaf,frac", [(1, 64, 0.5), (63, 64, 0.5), (64, 64, 0.5), (65, 64, 0.5), (128, 128, 0.5),
                                         (129, 128, 0.5), (700, 700, 0.5), (700, 97, 1.0), (701, 97, 0.3),
                                         (2001, 40, 0.66), (3003, 300, 0.9)])
def test_units_match_64_bit_solve(n, leaf, frac, lu):
    import torch
    from perf import cases
    for op in (1, 2, 3):
        case = {"kind": "ulv", "n": n, "leaf": leaf, "frac": frac, "frac_up": 0.5, "lu": lu, "op": op}
        x = cases.run(cases.prepare(case, 3)).clone()
        torch.cuda.synchronize()
        e = cases.exact(case, 3)
        assert float((x - e).norm() / e.norm()) < 1e-13, (n, leaf, lu, op)


def test_an_infinite_entry_reaches_only_what_depends_on_it():
    """Forward sweep of one node (the root, no Q): rows before an infinite right-hand side
    entry keep the values they have without it."""
    import torch
    from perf import cases
    case = {"kind": "ulv", "n": 150, "leaf": 150, "frac": 0.5, "frac_up": 0.5, "lu": False, "op": 1}
    s = cases.prepare(case, 5)
    clean = cases.run(s).clone()
    u = s["ulv"]
    k = 70                                     # second block of the permuted vector
    s["b"][int(u.fwd[k])] = float("inf")
    bad = cases.run(s).clone()
    torch.cuda.synchronize()
    inv = torch.from_numpy(u.bwd.astype("int64")).cuda()
    order = torch.empty_like(inv)
    order[inv] = torch.arange(150, device="cuda")          # x[i] = permuted[bwd[i]]
    assert torch.equal(clean[order][:k], bad[order][:k])
    assert not torch.isfinite(bad[order][k:]).all()


class _Kept:
    """The factors of one case, with the host arrays that create read kept for the test."""

    def __new__(cls, case, seed, change=None):
        from perf import cases

        class Ulv(cases._Ulv):
            def __setattr__(self, k, v):
                if not (k in ("hQ", "hL") and v is None):
                    super().__setattr__(k, v)

        u = Ulv(case, seed)
        if change:
            change(u)
        return u


@pytest.mark.parametrize("lu", [False, True])
def test_a_solve_right_after_create_sees_whole_factors(lu):
    """One node of 72 MB and three levels of small ones; the caller's arrays are overwritten as
    soon as create returns, and the first solve starts at once on the object's own stream."""
    import numpy as np
    import torch
    from h2pack_b200.h2pack import _dptr
    from perf import cases
    for n, leaf in ((3000, 3000), (3003, 60)):
        case = {"kind": "ulv", "n": n, "leaf": leaf, "frac": 0.6, "frac_up": 0.5, "lu": lu, "op": 3}
        b = np.random.default_rng(n).standard_normal(n)
        e = cases._Ulv(case, 8).solve(3, torch.from_numpy(b).cuda()).cpu().numpy()
        u = _Kept(case, 8)
        torch.cuda.synchronize()
        u.create()
        for a in u.hQ + u.hL:
            a.fill(np.nan)
        x = np.empty(n)
        assert u.lib.h2gpu_ulv_solve(u.handle, 3, _dptr(b), _dptr(x)) == 0
        assert np.linalg.norm(x - e) < 1e-13 * np.linalg.norm(e), (n, lu)


def _triangle(n, kind, lower, unit):
    """A triangular factor whose 64 x 64 diagonal blocks M are badly conditioned: "growth": entries -a
    beside a unit diagonal, || |M| |M^-1| || about (1 + a)^63 (a = 2^17: past the range of a
    double); "graded": rows scaled from 1 to 1e-14 within every block."""
    import numpy as np
    if kind == "graded":
        T = np.random.default_rng(n).standard_normal((n, n))
        np.fill_diagonal(T, 1.0)
        if not unit:
            T *= 10.0 ** (-14.0 * (np.arange(n) % 64) / 63.0)[:, None]
    else:
        T = np.full((n, n), -kind)
        np.fill_diagonal(T, 1.0)
    return np.tril(T) if lower else np.triu(T)


@pytest.mark.parametrize("lu", [False, True])
@pytest.mark.parametrize("kind", [0.05, 0.15, 0.3, 1.0, 4.0, 131072.0, "graded"])
@pytest.mark.parametrize("n", [50, 64, 200])
def test_ill_conditioned_diagonal_blocks(n, kind, lu):
    """The residual of a solve is that of substitution, whatever the blocks' conditioning: every
    row within n units of 1.1e-16 of |T| |x| (Higham, Accuracy and Stability, 8.1), here with
    a factor of two for the blocks that are solved with their inverse and one refinement (a residual
    of another 2e-18 of the block's right-hand side).  T x is formed in extended precision.  With
    a = 2^17 and whole numbers for unknowns substitution is exact, while the inverse overflows."""
    import numpy as np
    import torch
    from perf import cases
    case = {"kind": "ulv", "n": n, "leaf": n, "frac": 0.5, "frac_up": 0.5, "lu": lu, "op": 1}
    T0, T1 = _triangle(n, kind, True, lu), _triangle(n, kind, False, False)
    exact = kind == 131072.0

    def change(u):
        u.L[0] = torch.from_numpy(np.tril(T0, -1) + T1 if lu else T0).cuda()

    u = _Kept(case, 4, change)
    u.create()
    for op in (1, 2):
        T = T0 if op == 1 else (T1 if lu else T0.T)
        z = np.random.default_rng(7).integers(1, 9, n).astype(float)
        r = T @ (z if exact else z + np.random.default_rng(8).random(n))
        b = np.empty(n)
        b[u.fwd[u.p[0]] if lu and op == 1 else u.fwd] = r
        x = torch.empty(n, dtype=torch.float64, device="cuda")
        cases.run({"kind": "ulv", "ulv": u, "op": op, "b": torch.from_numpy(b).cuda(), "x": x})
        torch.cuda.synchronize()
        v = x.cpu().numpy()[u.fwd]
        if exact:
            assert np.array_equal(v, z), op
            continue
        W = T.astype(np.longdouble)
        res = np.abs(W @ v - r) / (np.abs(W) @ np.abs(v))
        assert float(res.max()) < 2 * n * 1.1e-16, (op, float(res.max()))


@pytest.mark.parametrize("lu", [False, True])
@pytest.mark.parametrize("n,leaf", [(40, 64), (700, 700), (2001, 40)])
def test_a_wait_that_runs_out_is_reported_once(n, leaf, lu):
    """One unit left out, so that the units which read its entries give up at the shortest limit: the
    check returns H2GPU_ERR_DEVICE, and the next solve is right (one unit alone waits for
    nothing)."""
    import torch
    from h2pack_b200 import _abi
    from perf import cases
    case = {"kind": "ulv", "n": n, "leaf": leaf, "frac": 0.6, "frac_up": 0.5, "lu": lu, "op": 3}
    s = cases.prepare(case, 3)
    u = s["ulv"]
    alone = n == 40 and not lu                  # LU: the unit that scatters waits for the block
    assert u.lib.h2gpu_ulv_wait_check(u.handle) == (_abi.H2GPU_OK if alone else -6)
    if not alone:
        assert b"bounded wait" in u.lib.h2gpu_last_error()
    x = cases.run(s).clone()
    torch.cuda.synchronize()
    e = cases.exact(case, 3)
    assert float((x - e).norm() / e.norm()) < 1e-13
    assert u.lib.h2gpu_ulv_solve(u.handle, 3, *[a.ctypes.data_as(cases.C.POINTER(cases.C.c_double))
                                                 for a in (s["b"].cpu().numpy(), x.cpu().numpy())]) == 0
