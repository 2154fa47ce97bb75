"""The steps of the fit kernels at the sizes where their work is divided: around one and two entries
per thread of the solving warps, the smallest class counts, score rows that stay in global memory,
against the restatement of the reference's solver."""
import numpy as np
import pytest

from libsdca_b200.synth import kernel_problem
from tests.test_fit_gpu import compare, dev, run_both
from tests.test_oracle_restatement import random_problem
from tests.util import stable_seed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle():
    from oracle import build_oracle, refapi
    build_oracle.build_restatement()
    return refapi.restatement()


def check_kernel(oracle, mod, objective, dtype, n, m, k, epochs, c=1.0, gamma=0.5):
    K, labels = kernel_problem(n=n, dim=8, m=m, seed=stable_seed(objective, n, m) % 1000, dtype=dtype)
    out = run_both(oracle, mod, objective, K, labels, m, True, dtype, c=c, gamma=gamma, k=k, max_epoch=epochs)
    compare(*out, 1e-9 if dtype == np.float64 else 2e-4, (objective, n, m, k))


def check_features(oracle, mod, objective, dtype, n, d, m, k, epochs, c=1.0, gamma=0.5, scale=1.0):
    rng = np.random.default_rng(stable_seed("features", objective, n, m))
    X, labels, _ = random_problem(rng, n, d, m, dtype, False)
    out = run_both(oracle, mod, objective, (X * scale).astype(dtype), labels, m, False, dtype, c=c, gamma=gamma,
                   k=k, max_epoch=epochs)
    compare(*out, 1e-9 if dtype == np.float64 else 2e-4, (objective, n, d, m, k))


@pytest.mark.parametrize("objective", ["l2_entropy", "l2_entropy_topk"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_entropic_steps(oracle, cuda_lib, objective, dtype):
    for n, m in ((70, 2), (65, 5), (130, 31), (200, 127), (200, 128), (200, 129), (150, 257)):
        k = 1 if objective == "l2_entropy" else min(3, m - 1)
        check_kernel(oracle, cuda_lib, objective, dtype, n, m, k, 4)
    # features scaled so that the top-k softmax step has one well-defined course
    for n, d, m in ((90, 7, 5), (150, 40, 129)):
        k = 1 if objective == "l2_entropy" else 2
        check_features(oracle, cuda_lib, objective, dtype, n, d, m, k, 4, c=0.1, scale=0.1)


def test_entropic_steps_with_rows_in_global_memory(oracle, cuda_lib):
    check_kernel(oracle, cuda_lib, "l2_entropy", np.float64, 130, 600, 1, 2)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kernel", [False, True])
def test_multilabel_entropic_steps(oracle, cuda_lib, dtype, kernel):
    from oracle.refapi import OBJECTIVES as IDS
    rng = np.random.default_rng(stable_seed("multilabel entropic", str(dtype), kernel))
    for n, d, m in ((70, 6, 3), (140, 12, 33), (200, 20, 128), (140, 12, 161)):
        X, labels, offsets = random_problem(rng, n, d, m, dtype, True)
        data = (X.astype(np.float64) @ X.astype(np.float64).T).astype(dtype) if kernel else X
        kw = dict(c=0.9, gamma=0.7, k=1, epsilon=1e-3, max_epoch=4, eval_epoch=2)
        A_ref = np.zeros((n, m), dtype=dtype)
        W_ref = np.zeros((m, d), dtype=dtype)
        r = oracle.fit("l2_multilabel_entropy", data, A_ref, labels, W=None if kernel else W_ref, kernel=kernel,
                       offsets=offsets, **kw)
        A, W = dev(np.zeros((n, m), dtype=dtype)), None if kernel else dev(np.zeros((m, d), dtype=dtype))
        g = cuda_lib.fit_(IDS["l2_multilabel_entropy"], dev(data), dev(labels), A, W=W, kernel=kernel,
                          offsets=dev(offsets), **kw)
        compare(r, g, A_ref, W_ref, A.cpu().numpy(), None if kernel else W.cpu().numpy(),
                1e-9 if dtype == np.float64 else 2e-4, (n, m, kernel))


@pytest.mark.parametrize("objective", ["l2_hinge_topk", "l2_hinge_topk_smooth", "l2_topk_hinge", "l2_topk_hinge_smooth"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_hinge_steps(oracle, cuda_lib, objective, dtype):
    """Rows in 2, 4 and 8 registers per lane, k up to all but one of the other classes and beyond,
    and features with far-off scores, whose steps end at <1, x> = c."""
    for n, m, k in ((70, 3, 1), (70, 3, 2), (65, 6, 4), (130, 64, 5), (130, 65, 5), (200, 128, 10), (200, 129, 3),
                    (150, 256, 32), (150, 256, 33)):
        check_kernel(oracle, cuda_lib, objective, dtype, n, m, k, 4)
    for n, d, m, k in ((90, 7, 5, 2), (300, 40, 64, 5), (150, 20, 129, 3)):
        check_features(oracle, cuda_lib, objective, dtype, n, d, m, k, 3, c=0.05)
        check_features(oracle, cuda_lib, objective, dtype, n, d, m, k, 3, c=1.0, scale=0.2)


@pytest.mark.parametrize("objective", ["l2_multilabel_hinge", "l2_multilabel_hinge_smooth"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kernel", [False, True])
def test_multilabel_hinge_steps(oracle, cuda_lib, objective, dtype, kernel):
    """Rows in 2, 4 and 8 registers per lane and the general step beyond, steps that end in either
    phase of the projection (small c: both blocks reach it)."""
    from oracle.refapi import OBJECTIVES as IDS
    rng = np.random.default_rng(stable_seed("multilabel hinge", objective, str(dtype), kernel))
    for n, d, m, c in ((70, 6, 3, 0.9), (70, 6, 3, 0.01), (140, 12, 33, 0.9), (140, 12, 64, 0.01), (140, 12, 65, 0.9),
                       (200, 20, 128, 0.5), (140, 12, 129, 0.9), (140, 12, 256, 0.02), (140, 12, 257, 0.9)):
        X, labels, offsets = random_problem(rng, n, d, m, dtype, True)
        data = (X.astype(np.float64) @ X.astype(np.float64).T).astype(dtype) if kernel else X
        kw = dict(c=c, gamma=0.7, k=1, epsilon=1e-4, max_epoch=4, eval_epoch=2)
        A_ref, W_ref = np.zeros((n, m), dtype=dtype), np.zeros((m, d), dtype=dtype)
        r = oracle.fit(objective, data, A_ref, labels, W=None if kernel else W_ref, kernel=kernel, offsets=offsets,
                       **kw)
        A, W = dev(np.zeros((n, m), dtype=dtype)), None if kernel else dev(np.zeros((m, d), dtype=dtype))
        g = cuda_lib.fit_(IDS[objective], dev(data), dev(labels), A, W=W, kernel=kernel, offsets=dev(offsets), **kw)
        compare(r, g, A_ref, W_ref, A.cpu().numpy(), None if kernel else W.cpu().numpy(),
                1e-9 if dtype == np.float64 else 2e-4, (n, m, c, kernel))


@pytest.mark.parametrize("objective", ["l2_topk_hinge", "l2_hinge_topk", "l2_entropy"])
@pytest.mark.parametrize("dtype,classes", [(np.float64, range(342, 350)), (np.float32, range(354, 362))])
def test_class_counts_at_which_the_score_rows_leave_shared_memory(oracle, cuda_lib, objective, dtype, classes):
    for m in classes:
        check_kernel(oracle, cuda_lib, objective, dtype, 70, m, 3 if "topk" in objective else 1, 1)


def test_class_counts_beyond_shared_memory_are_refused(cuda_lib):
    """Even one score row has to fit: up to there a fit runs, from there on it says so."""
    import torch
    refused = []
    for m in (3400, 3475, 3485, 3500, 3512, 3520, 3600):
        K = torch.eye(4, dtype=torch.float64, device="cuda")
        A = torch.zeros(4, m, dtype=torch.float64, device="cuda")
        try:
            cuda_lib.fit_("msvm", K, torch.arange(4, device="cuda"), A, kernel=True, max_epoch=1, eval_epoch=1)
            refused.append(False)
            assert bool((A.sum(dim=1).abs() < 1e-12).all()) and bool(A.any())
        except cuda_lib.SdcabError as error:
            assert "too_large" in str(error), error
            refused.append(True)
    assert refused == sorted(refused) and not refused[0] and refused[-1]


@pytest.mark.parametrize("multilabel", [False, True])
def test_many_held_out_sets(cuda_lib, multilabel):
    """Host arrays with more held-out sets than anybody would expect, each one's records its own."""
    rng = np.random.default_rng(stable_seed("held out", multilabel))
    n, d, m = 40, 6, 5
    X, labels, offsets = random_problem(rng, n, d, m, np.float64, multilabel)
    tests = []
    for i in range(20):
        Xi, li, oi = random_problem(rng, 10 + i, d, m, np.float64, multilabel)
        tests.append((Xi, li, oi) if multilabel else (Xi, li))
    A, W = np.zeros((n, m)), np.zeros((m, d))
    objective = "mlsvm" if multilabel else "msvm"
    out = cuda_lib.fit_(objective, X, labels, A, W=W, offsets=offsets, max_epoch=2, eval_epoch=1, tests=tests)
    assert len(out["tests"]) == len(tests)
    for got, t in zip(out["tests"], tests):
        want = cuda_lib.evaluate(objective, t[0], t[1], W=W, offsets=t[2] if multilabel else None, is_train=False)
        assert abs(got["primal_loss"][-1] - want["primal_loss"]) <= 1e-12 * max(1.0, want["primal_loss"])
