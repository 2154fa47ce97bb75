"""The softmax loss with the score row in registers, at the sizes where the number of entries per
lane changes and at one to just over 32 examples a warp, against the restatement of the reference
and against the general loss kernel."""
import numpy as np
import pytest

from tests.test_oracle_restatement import random_problem
from tests.util import stable_seed

pytestmark = pytest.mark.gpu


def dev(x):
    import torch
    return None if x is None else torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kernel", [False, True])
@pytest.mark.parametrize("precision", ["double", "float"])
def test_softmax_loss(cuda_lib, dtype, kernel, precision):
    from libsdca_b200 import binding as b
    from oracle import build_oracle, refapi
    build_oracle.build_restatement()
    oracle = refapi.restatement()
    rng = np.random.default_rng(stable_seed("softmax loss", str(dtype), kernel))
    for n, d, m in ((3, 4, 2), (50, 6, 31), (70, 6, 32), (70, 6, 33), (200, 9, 101), (90, 8, 128), (90, 8, 129),
                    (80, 8, 256), (80, 8, 257), (60, 8, 1000), (40, 8, 1024), (40, 8, 1025)):
        X, labels, _ = random_problem(rng, n, d, m, dtype, False)
        c = 0.7
        # a feasible dual: -c p for the other classes, their sum for the label
        p = rng.dirichlet(np.ones(m), size=n) * c
        A = -p
        A[np.arange(n), labels] = 0
        A[np.arange(n), labels] = -A.sum(axis=1)
        A = A.astype(dtype)
        W = None if kernel else (A.T @ X).astype(dtype)
        data = (X @ X.T).astype(dtype) if kernel else X
        r = oracle.evaluate("l2_entropy", data, A, labels, W=W, kernel=kernel, c=c)
        args = (0, dev(data), dev(labels))
        kw = dict(A=dev(A), W=dev(W), kernel=kernel, c=c, precision=precision)
        got = cuda_lib.evaluate(*args, **kw)
        # sums of n m terms of order one, rounded at the type's precision
        eps = np.finfo(np.float32 if dtype == np.float32 or precision == "float" else np.float64).eps
        tol = 16 * eps * np.sqrt(n * m)
        try:
            b.test_set("loss_general", 1)
            general = cuda_lib.evaluate(*args, **kw)
        finally:
            b.test_set("loss_general", 0)
        for f in ("primal_loss", "dual_loss", "primal", "dual"):
            assert abs(got[f] - r[f]) <= tol * max(1.0, abs(r[f])), (n, m, f, got[f], r[f])
            assert abs(got[f] - general[f]) <= tol * max(1.0, abs(general[f])), (n, m, f)
        assert np.array_equal(got["accuracy"], general["accuracy"]), (n, m)
        held_out = cuda_lib.evaluate(*args, **dict(kw, is_train=False))
        assert abs(held_out["primal_loss"] - got["primal_loss"]) <= tol * max(1.0, abs(got["primal_loss"]))


def test_softmax_loss_of_many_examples_repeats_bit_for_bit(cuda_lib):
    """More than 32 examples for every warp of the launch, twice."""
    rng = np.random.default_rng(12)
    X = rng.standard_normal((400000, 3))
    W = rng.standard_normal((5, 3))
    labels = rng.integers(0, 5, len(X))
    first = cuda_lib.evaluate(0, dev(X), dev(labels), W=dev(W), is_train=False)
    again = cuda_lib.evaluate(0, dev(X), dev(labels), W=dev(W), is_train=False)
    assert first["primal_loss"] == again["primal_loss"]
    scores = X @ W.T
    top = scores.max(axis=1)
    exact = (top + np.log(np.exp(scores - top[:, None]).sum(axis=1)) - scores[np.arange(len(X)), labels]).sum()
    assert abs(first["primal_loss"] - exact) <= 1e-12 * abs(exact)


def guarded_sums(mod, X, labels, W, dtype, precision):
    """One evaluation in a workspace of exactly the required size with a pattern behind it: the sums, and
    whether the pattern is still there."""
    import ctypes as C

    import torch
    from libsdca_b200 import binding as b
    m = W.shape[0]
    obj = b.make_objective(0, precision=precision)
    problem = b.make_problem(X, labels, W=W, is_train=False)
    suffix = "f32" if dtype == np.float32 else "f64"
    query = mod.lib()["sdcab_eval_workspace_bytes"]
    query.restype = C.c_size_t
    need = query(C.c_int64(X.shape[0]), C.c_int64(m), C.c_int64(np.dtype(dtype).itemsize))
    guard = 16384
    work = torch.full((need + guard,), 0x5a, dtype=torch.uint8, device="cuda")
    sums = torch.zeros(8 + m, dtype=torch.float64, device="cuda")
    b.eval_sums_(obj, problem, sums, suffix, work, need)
    return sums.cpu().numpy(), bool((work[need:] == 0x5a).all())


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("precision", ["double", "float"])
def test_softmax_loss_of_infinite_scores(cuda_lib, dtype, precision):
    """A label's score of -inf, and rows of infinities: the ranks and the loss are those of the general kernel,
    and nothing is written past the histogram."""
    from libsdca_b200 import binding as b
    rng = np.random.default_rng(stable_seed("infinite", str(dtype), precision))
    for m in (2, 20, 32, 101, 128, 200, 256, 257, 300, 600, 1000, 1024):
        n = 12
        scores = rng.standard_normal((m, n))
        labels = rng.integers(0, m, n)
        scores[labels[0], 0] = -np.inf
        scores[labels[1], 1] = scores[(labels[1] + 1) % m, 1] = -np.inf
        scores[:, 2] = -np.inf
        scores[labels[3], 3] = np.inf
        scores[(labels[4] + 1) % m, 4] = np.inf
        scores[:, 5] = np.inf
        scores[labels[6], 6] = np.nan
        scores[(labels[7] + 1) % m, 7] = np.nan
        # one feature and one example at a time: in a product of several, 0 * inf would reach other scores
        for e in range(n):
            W = dev(scores[:, e:e + 1].astype(dtype))
            args = (cuda_lib, dev(np.ones((1, 1), dtype=dtype)), dev(labels[e:e + 1]), W, dtype, precision)
            got, kept = guarded_sums(*args)
            try:
                b.test_set("loss_general", 1)
                general, _ = guarded_sums(*args)
            finally:
                b.test_set("loss_general", 0)
            assert kept, (m, e)
            assert np.array_equal(got[8:], general[8:]) and got[8:].sum() == 1, (m, e)
            assert got[6] == 0, (m, e)
            assert np.allclose(got[0], general[0], rtol=1e-5 if "float" in (precision, np.dtype(dtype).name[:5]) else 1e-12,
                               equal_nan=True), (m, e, got[0], general[0])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("precision", ["double", "float"])
def test_softmax_loss_of_confident_models(cuda_lib, dtype, precision):
    """Losses far below one: what is left of an example's loss is the small sum next to the one of its
    own class."""
    rng = np.random.default_rng(stable_seed("confident", str(dtype), precision))
    for m, margin in ((2, 40.0), (31, 25.0), (101, 20.0), (129, 30.0), (300, 12.0), (1000, 20.0)):
        W = (-margin - rng.uniform(0, 2, (m, 1))).astype(dtype)
        W[m // 2] = 0
        labels = np.full(50, m // 2)
        got = cuda_lib.evaluate(0, dev(np.ones((50, 1), dtype=dtype)), dev(labels), W=dev(W), is_train=False,
                                precision=precision)
        loss = 50 * np.log1p(np.exp(np.delete(W, m // 2).astype(np.float64)).sum())
        # m exponentials, 4 eps each, and their sum in another order
        eps = np.finfo(np.float32 if dtype == np.float32 or precision == "float" else np.float64).eps
        assert abs(got["primal_loss"] / loss - 1) <= 16 * eps + 1e-14, (m, margin)
