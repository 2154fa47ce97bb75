"""Calls of several host threads at the same time."""
import pytest

pytestmark = pytest.mark.gpu


def test_calls_of_several_threads(cuda_lib):
    """Rows of different lengths at the same time, whose launches need different amounts of shared memory."""
    import threading

    import torch
    rows = {m: torch.randn(3000 * m, m, dtype=torch.float64, device="cuda") for m in (49, 64)}
    want = {m: cuda_lib.prox(a, "topk_cone", k=3) for m, a in rows.items()}
    failures = []

    def work(m):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                out = torch.empty_like(rows[m])
                for _ in range(400):
                    cuda_lib.prox_to(rows[m], out, "topk_cone", k=3)
                torch.cuda.current_stream().synchronize()
                assert torch.equal(out, want[m]), m
        except Exception as error:      # noqa: BLE001 -- reported by the main thread
            failures.append((m, error))

    threads = [threading.Thread(target=work, args=(m,)) for m in (49, 64, 49, 64)]
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
