"""The row kernels at the edges of what each takes: lengths that no vector width divides, rows that
do not start on 16-byte boundaries, rows of a whole block, against the restatement of the reference."""
import numpy as np
import pytest

from tests.util import float_precision_ok, random_opts, regime, scaled_error, stable_seed, tolerance

pytestmark = pytest.mark.gpu

KINDS = ("normal", "pos", "neg", "mixed", "ties")
TYPES = [(np.float64, "double"), (np.float32, "double"), (np.float32, "float")]


@pytest.fixture(scope="module")
def oracle():
    from oracle import build_oracle, refapi
    build_oracle.build_restatement()
    return refapi.restatement()


def run_dev(mod, name, a, offset, **kw):
    """The projection of `a` laid out `offset` elements behind a 16-byte boundary."""
    import torch
    flat = torch.empty(a.size + 4, dtype=torch.from_numpy(a).dtype, device="cuda")
    t = flat[offset:offset + a.size].view(a.shape)
    t.copy_(torch.from_numpy(a))
    mod.prox_(t, name, **kw)
    torch.cuda.synchronize()
    return t.cpu().numpy()


def check(oracle, cuda_lib, name, a, precision, offset=0, **kw):
    x = run_dev(cuda_lib, name, a, offset, precision=precision, **kw)
    x_ref = oracle.prox(name, a, result=precision, **kw)
    tol = tolerance(a.dtype, precision, a.shape[1])
    if precision == "double":
        err = scaled_error(x, x_ref, a).max()
        assert err <= tol, (name, a.shape, kw, err)
    else:
        ok, err = float_precision_ok(x, x_ref, oracle.prox(name, a, result="double", **kw), a, tol)
        assert ok, (name, a.shape, kw, err)


@pytest.mark.parametrize("name", ["knapsack_eq", "knapsack_le", "knapsack_le_biased", "topk_simplex",
                                  "topk_simplex_biased", "topk_cone", "topk_cone_biased", "entropy",
                                  "topk_entropy"])
@pytest.mark.parametrize("dtype,precision", TYPES)
def test_rows_off_the_vector_grid(oracle, cuda_lib, name, dtype, precision):
    """Element-wise register rows (with float thresholds the general kernel, the same sizes)."""
    rng = np.random.default_rng(stable_seed("off-grid", name, str(dtype), precision))
    # one past / one short of each number of elements per lane, and even lengths on an odd base
    for m, offset in ((9, 0), (31, 0), (33, 1), (129, 0), (255, 0), (256, 1), (257, 0), (511, 0), (512, 1),
                      (513, 0), (999, 0), (1000, 1), (1023, 0)):
        kinds = KINDS if m < 300 else ("normal", "ties")
        for kind in kinds:
            a = regime(rng, 21, m, dtype, kind)
            check(oracle, cuda_lib, name, a, precision, offset, **random_opts(rng, name, m))


@pytest.mark.parametrize("name", ["entropy", "topk_entropy"])
def test_grouped_entropic_rows_off_the_vector_grid(oracle, cuda_lib, name):
    """Enough rows for the kernel that batches the closed forms of up to 32 rows."""
    import torch
    blocks = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(stable_seed("grouped off-grid", name))
    for m, offset in ((33, 0), (63, 0), (64, 1), (255, 0), (257, 0)):
        a = (2 * rng.standard_normal((12 * blocks + 5, m))).astype(np.float32)
        kw = dict(k=min(10, m)) if name == "topk_entropy" else dict(hi=1.0, rhs=1.0)
        x = run_dev(cuda_lib, name, a, offset, **kw)
        rows = rng.permutation(len(a))[:400]
        x_ref = oracle.prox(name, a[rows], **kw)
        assert scaled_error(x[rows], x_ref, a[rows]).max() <= 1e-5, (name, m)
        assert np.abs(x.sum(axis=1, dtype=np.float64)).max() <= 1 + 1e-5


LONG = ["knapsack_eq", "knapsack_le", "knapsack_le_biased", "topk_simplex", "topk_simplex_biased", "topk_cone"]


@pytest.mark.parametrize("name", LONG)
@pytest.mark.parametrize("dtype,precision", TYPES)
def test_long_rows(oracle, cuda_lib, name, dtype, precision):
    """Rows above the register kernels' limit, at the sizes where the block grows, where the copy no
    longer fits shared memory, and off the vector grid.  Doubles above 1024 entries and float thresholds
    are the general kernel's at any length."""
    item = np.dtype(dtype).itemsize
    rng = np.random.default_rng(stable_seed("long", name, str(dtype), precision))
    sizes = [(4096 // item + 1, 0), (1000 if item == 8 else 1027, 1), (1024 if item == 8 else 4095, 0), (1025, 1),
             (2048, 0), (16384 // item, 1), (16384 // item + 1, 0),
             (57344 // item, 0), (57344 // item + 3, 1), (240000 // item, 1)]
    for m, offset in sizes:
        for kind in KINDS if m < 4000 else ("normal", "ties"):
            a = regime(rng, 7 if m < 10000 else 3, m, dtype, kind)
            check(oracle, cuda_lib, name, a, precision, offset, **random_opts(rng, name, m))


@pytest.mark.parametrize("name", LONG)
@pytest.mark.parametrize("dtype,m", [(np.float64, 1000), (np.float32, 3000)])
def test_long_rows_with_crowded_tops(oracle, cuda_lib, name, dtype, m):
    """More candidates than one warp takes, than the block keeps, all entries equal, one dominating
    entry: the same answers as the general routine gives."""
    rng = np.random.default_rng(stable_seed("crowded", name))
    rows = [1e-3 * rng.standard_normal(m), 1e-2 * rng.standard_normal(m), 0.1 * rng.standard_normal(m),
            np.full(m, 0.25), np.full(m, -1.0), np.zeros(m), rng.standard_normal(m)]
    rows[6][17] = 50.0
    a = np.stack(rows).astype(dtype)
    for kw in (dict(), dict(rhs=4.0)) if name != "topk_cone" else (dict(),):
        k = dict(k=5) if name.startswith("topk") else {}
        check(oracle, cuda_lib, name, a, "double", **kw, **k)


@pytest.mark.parametrize("name", LONG)
@pytest.mark.parametrize("dtype,m", [(np.float64, 513), (np.float64, 1024), (np.float32, 1025), (np.float32, 5000)])
def test_long_rows_repeat_bit_for_bit(cuda_lib, name, dtype, m):
    """Few candidates and many: the order in which a block's threads find them must not show."""
    import torch
    rng = np.random.default_rng(8)
    for scale in (1.0, 0.05):
        a = torch.from_numpy((scale * rng.standard_normal((4000, m))).astype(dtype)).cuda()
        kw = dict(k=5) if name.startswith("topk") else {}
        first = cuda_lib.prox(a, name, **kw)
        for _ in range(6):
            assert torch.equal(first, cuda_lib.prox(a, name, **kw)), (name, m, scale)


@pytest.mark.parametrize("name", ["knapsack_eq", "knapsack_le", "knapsack_le_biased", "topk_simplex",
                                  "topk_simplex_biased", "topk_cone", "topk_cone_biased", "entropy",
                                  "topk_entropy"])
@pytest.mark.parametrize("dtype,precision", TYPES)
def test_many_short_rows(oracle, cuda_lib, name, dtype, precision):
    """One thread per row: the lengths around the limits of the operators, the first row count that
    takes the kernel and the last that does not, a last block that is not full.  Float thresholds keep
    one warp per row."""
    import torch
    rng = np.random.default_rng(stable_seed("short", name, str(dtype), precision))
    for m, n, offset in ((1, 3000, 0), (2, 6001, 1), (7, 21127, 0), (8, 23999, 0), (10, 30005, 1), (31, 93100, 0),
                         (32, 96001, 1), (33, 99000, 0), (40, 120003, 0), (41, 123000, 1), (48, 144001, 0),
                         (49, 147000, 0), (64, 192002, 1), (65, 195000, 0)):
        rows = np.concatenate([regime(rng, 20, m, dtype, kind) for kind in KINDS])
        kw = random_opts(rng, name, m)
        base = torch.from_numpy(rows).cuda()
        flat = torch.empty(n * m + 4, dtype=base.dtype, device="cuda")
        t = flat[offset:offset + n * m].view(n, m)
        which = torch.arange(n, device="cuda") % len(rows)
        t.copy_(base[which])
        cuda_lib.prox_(t, name, precision=precision, **kw)
        x = t[:len(rows)].cpu().numpy()
        tol = tolerance(dtype, precision, m)
        # equal rows, equal results up to the order of the sums
        scale = base.double().abs().amax(dim=1, keepdim=True).clamp(min=1)[which]
        assert float(((t.double() - t[:len(rows)].double()[which]) / scale).abs().max()) <= tol, (name, m, kw)
        x_ref = oracle.prox(name, rows, result=precision, **kw)
        if precision == "double":
            assert scaled_error(x, x_ref, rows).max() <= tol, (name, m, kw)
        else:
            ok, err = float_precision_ok(x, x_ref, oracle.prox(name, rows, result="double", **kw), rows, tol)
            assert ok, (name, m, kw, err)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_biased_topk_entropy_of_large_entries(oracle, cuda_lib, dtype):
    """Rows in the hundreds and thousands, where the iteration for some sizes of U runs to s = 0 with t
    far above the entries, and the reference accepts that."""
    rng = np.random.default_rng(stable_seed("large entries", str(dtype)))
    for m, k, alpha in ((15, 12, 4.0), (18, 12, 1.9), (22, 12, 3.6), (16, 5, 5.0), (40, 12, 4.3)):
        a = (rng.standard_normal((6000, m)) * 10.0 ** rng.uniform(1, 4, (6000, 1))).astype(dtype)
        kw = dict(k=k, alpha=alpha)
        x = run_dev(cuda_lib, "topk_entropy_biased", a, 0, **kw)
        # an entry's last bit is 1e-16 (double) or 6e-8 (float) of 1e4, and t and the outputs move with it
        tol = 1e-9 if dtype == np.float64 else 1e-2
        assert np.abs(x - oracle.prox("topk_entropy_biased", a, **kw)).max() <= tol, (m, k, alpha)
