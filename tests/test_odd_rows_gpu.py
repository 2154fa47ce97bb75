"""Rows that hold NaN, infinities or the lowest value of their type, through every kernel that takes rows,
against the restatement of the reference."""
import numpy as np
import pytest

from tests.test_row_kernels_gpu import LONG, oracle, run_dev  # noqa: F401
from tests.util import scaled_error, stable_seed, tolerance

pytestmark = pytest.mark.gpu


def rows_repeat(t, rows, tol):
    """Rows r, r + rows, r + 2 rows, ... agree (up to the order of the sums over candidates)."""
    import torch
    first = t[:rows][torch.arange(len(t), device=t.device) % rows]
    return bool(torch.isclose(t, first, rtol=10 * tol, atol=10 * tol).all())


@pytest.mark.parametrize("name", LONG)
@pytest.mark.parametrize("dtype,m", [(np.float64, 1000), (np.float32, 3000)])
def test_long_rows_that_are_not_finite(oracle, cuda_lib, name, dtype, m):
    """Infinities and NaN are the general routine's: the restatement's answer, except that its
    knapsack_le_biased depends on the order of the entries then."""
    rng = np.random.default_rng(stable_seed("not finite", name, m))
    a = rng.standard_normal((6, m)).astype(dtype)
    a[0, 5] = np.inf
    a[1, [7, m - 1]] = np.inf
    a[2, 11] = np.nan
    a[3, :m // 2] = -np.inf
    a[4, 3], a[4, 4] = np.inf, -np.inf
    keep = [0, 1, 5] if name == "knapsack_le_biased" else range(6)
    kw = dict(k=5) if name.startswith("topk") else {}
    x, x_ref = run_dev(cuda_lib, name, a, 0, **kw), oracle.prox(name, a, **kw)
    for r in keep:
        assert np.abs(x[r].astype(np.float64) - x_ref[r]).max() <= tolerance(dtype, "double", m) * 5, (name, r)


def odd_rows(rng, dtype, m):
    """Rows with NaN and infinities, an ordinary one between each two of them."""
    a = rng.standard_normal((23, m)).astype(dtype)
    odd = a[1::2]
    odd[0, 0] = np.nan
    odd[1, m // 2] = np.nan
    odd[2, [1, m - 1]] = np.nan
    odd[3] = np.nan
    odd[4, m // 3] = np.inf
    odd[5, [2, m - 2]] = np.inf
    odd[6, m // 2:] = -np.inf
    odd[7] = -np.inf
    odd[8, 0], odd[8, 1] = np.inf, -np.inf
    odd[9, 3], odd[9, 4] = np.nan, np.inf
    odd[10, ::2] = np.finfo(dtype).min
    return a


@pytest.mark.parametrize("name", ["knapsack_eq", "knapsack_le", "knapsack_le_biased", "topk_simplex",
                                  "topk_simplex_biased", "topk_cone", "topk_cone_biased", "entropy", "entropy_norm",
                                  "topk_entropy", "topk_entropy_biased", "two_simplex"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_rows_that_are_not_finite(oracle, cuda_lib, name, dtype):
    """Whatever such a row holds, its search ends, gives numbers, and leaves its neighbours alone: one
    thread per row, registers on and off the vector grid, a block per row, one warp per row."""
    import torch
    rng = np.random.default_rng(stable_seed("odd rows", name, str(dtype)))
    for m, n in ((10, 30000), (31, 93000), (40, 120000), (40, 23), (100, 23), (101, 23), (300, 23), (513, 23),
                 (1000, 23), (1023, 23), (1500, 23)):
        a = odd_rows(rng, dtype, m)
        for kw in [dict(k=1), dict(k=3)] if name.startswith("topk") else [dict(p=5)] if name == "two_simplex" else [{}]:
            t = torch.from_numpy(a).cuda()[torch.arange(n, device="cuda") % len(a)]
            x = cuda_lib.prox(t, name, **kw)
            assert rows_repeat(x, len(a), tolerance(dtype, "double", m)), (name, m, kw)
            x = x[:len(a)].cpu().numpy()
            assert not np.isnan(x).any(), (name, m, kw)
            x_ref = oracle.prox(name, a[0::2], **kw)
            assert scaled_error(x[0::2], x_ref, a[0::2]).max() <= tolerance(dtype, "double", m), (name, m, kw)


@pytest.mark.parametrize("objective", ["msvm", "msvm_smooth", "topk_hinge_alpha", "topk_hinge_beta", "softmax",
                                       "l2_entropy_topk", "mlsvm", "mlsvm_smooth", "mlsoftmax"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_evaluation_of_scores_that_are_nan(cuda_lib, objective, dtype):
    """The loss of a model that has diverged on one example is NaN, its evaluation ends, and the ranks
    are those of the scores that are numbers."""
    import torch
    rng = np.random.default_rng(stable_seed("nan scores", objective, str(dtype)))
    multilabel = objective.startswith("ml")
    for gamma in (0.0, 1.0) if "topk_hinge" in objective else (1.0 if "smooth" in objective else 0.0,):
        for n, d, m in ((70, 5, 20), (70, 33, 100), (70, 40, 300), (40, 40, 1100)):
            X = rng.standard_normal((n, d)).astype(dtype)
            X[n // 2, 1] = np.nan
            W = rng.standard_normal((m, d)).astype(dtype)
            labels = rng.integers(0, m, n)
            put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).cuda()       # noqa: E731
            offsets = put(np.arange(n + 1)) if multilabel else None
            kw = dict(k=3 if "topk" in objective else 1, gamma=gamma, offsets=offsets, is_train=False)
            got = cuda_lib.evaluate(objective, put(X), put(labels), W=put(W), **kw)
            good = np.delete(np.arange(n), n // 2)
            if multilabel:
                kw["offsets"] = put(np.arange(n))
            rest = cuda_lib.evaluate(objective, put(X[good]), put(labels[good]), W=put(W), **kw)
            assert np.isnan(got["primal_loss"]) or got["primal_loss"] >= rest["primal_loss"] * (1 - 1e-5), (n, m)
            if not multilabel:
                # no class scores at least as high as NaN: the example counts as rank 0
                want = (rest["accuracy"] * (n - 1) + 1) / n
                assert np.abs(got["accuracy"] - want).max() <= 1e-9, (n, m)


# Rows of which a part is ruled out by a very small value.  The answer is the projection of the other
# entries and 0 for these: the operators' supports lie near the top of a row.
MASKED = {"knapsack_eq": {}, "knapsack_le": {}, "knapsack_le_biased": dict(rho=0.1), "topk_simplex": dict(k=3),
          "topk_simplex_biased": dict(k=3, rho=0.01), "topk_cone": dict(k=3), "entropy": {}, "topk_entropy": dict(k=3)}


@pytest.mark.parametrize("name", MASKED)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_masked_entries(oracle, cuda_lib, name, dtype):
    import torch
    rng = np.random.default_rng(stable_seed("masked", name, str(dtype)))
    lowest = float(np.finfo(dtype).min)
    # one thread per row (on and off the vector grid), registers (on and off), a block per row
    for m, n, offset, values in ((10, 30000, 0, (-np.inf, lowest, -1e30)), (31, 93000, 1, (-np.inf, lowest, -1e30)),
                                 (32, 96000, 0, (-np.inf, lowest, -1e30)), (40, 120000, 0, (-np.inf, lowest, -1e30)),
                                 (100, 60, 0, (-np.inf, lowest, -1e30)), (101, 60, 0, (-np.inf, lowest, -1e30)),
                                 (300, 60, 1, (-np.inf, lowest, -1e30)), (1000, 60, 0, (lowest, -1e30)),
                                 (1025, 60, 0, (lowest, -1e30))):
        if m == 1025 and dtype == np.float64:
            continue                     # rows of doubles this long are the general kernel's
        for value in values:
            rows, kept = 60, m - max(3, m // 3)
            a = rng.standard_normal((rows, m)).astype(dtype) + 1
            where = rng.permuted(np.tile(np.arange(m), (rows, 1)), axis=1)
            keep, drop = np.sort(where[:, :kept], axis=1), where[:, kept:]
            part = np.take_along_axis(a, keep, axis=1)
            np.put_along_axis(a, drop, dtype(value), axis=1)
            flat = torch.empty(n * m + 4, dtype=torch.from_numpy(a).dtype, device="cuda")
            t = flat[offset:offset + n * m].view(n, m)
            t.copy_(torch.from_numpy(a).cuda()[torch.arange(n, device="cuda") % rows])
            cuda_lib.prox_(t, name, **MASKED[name])
            x = t[:rows].cpu().numpy()
            assert rows_repeat(t, rows, tolerance(dtype, "double", m)), (name, m, value)
            assert not np.take_along_axis(x, drop, axis=1).any(), (name, m, value)
            err = scaled_error(np.take_along_axis(x, keep, axis=1), oracle.prox(name, part, **MASKED[name]), part).max()
            assert err <= tolerance(dtype, "double", m), (name, m, value, err)
