"""Kept workspace and side streams that another stream's queue still needs hold nobody up: an operator on a second stream
finishes while the first stream is busy, and both give the results they give alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,N,n", [(torch.float64, 32, 3), (torch.float32, 48, 4)])
def test_second_stream_does_not_wait(dtype, N, n):
    from test_gpu_kept_workspace import compute, plan_of
    from gato_gb300.scf import release_workspace
    release_workspace()   # other tests' buffers: room for this one's
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    plans = {s: plan_of(N, dtype, n) for s in (a, b)}
    want = {}
    for s in (a, b, a, b):   # allocates what each stream keeps; the operators' buffers go back
        with torch.cuda.stream(s):
            want[s] = compute(N, n, dtype, 1, plans[s])
        torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(2_000_000_000)   # about a second
        first = compute(N, n, dtype, 1, plans[a])
    with torch.cuda.stream(b):
        second = compute(N, n, dtype, 1, plans[b])
        b.synchronize()
    busy = not a.query()
    torch.cuda.synchronize()
    for got, s in ((first, a), (second, b)):
        assert torch.equal(got[0], want[s][0]) and torch.equal(got[1], want[s][1])
    assert busy
