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
