"""Operator workspace kept from one operator to the next: same results whatever stream, thread or size had
the buffer before, and after a capture or a failed call. The comparison is exact: the same kernels run on
the same inputs."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def inputs(N, n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.rand(n, N, N, N, generator=g, dtype=torch.float64, device="cuda").to(dtype)
    return f, torch.rand(N, N, N, generator=g, dtype=torch.float64, device="cuda").to(dtype)


def compute(N, n, dtype, seed, plan):
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator
    f, V = inputs(N, n, dtype, seed)
    op = Operator(Grid3D(N, 0.25 * N), dtype, 4)
    op.set_potential(V)
    op.set_exchange(plan, f)
    return op.energy_terms(V), op.apply_block()


def plan_of(N, dtype, n):
    from gato_gb300.scf import pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    return PoissonPlan(N, 0.25, 0.125, dtype, pair_fields(n))


def test_streams_sizes_and_threads():
    cases = [(24, 3, torch.float64, 1), (48, 4, torch.float32, 2), (32, 2, torch.float64, 3), (24, 3, torch.float32, 4)]
    plans = [plan_of(N, dt, n) for N, n, dt, _ in cases]
    want = []
    for c, p in zip(cases, plans):
        want.append(compute(*c, p))
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    for rep in range(6):   # operators made and dropped back to back, no synchronisation in between
        got = []
        for k in range(len(cases)):
            i = (k * (rep % 3 + 1) + rep) % len(cases)
            with torch.cuda.stream(streams[i]):
                got.append((i, compute(*cases[i], plans[i])))
        torch.cuda.synchronize()
        for i, (e, b) in got:
            assert torch.equal(e, want[i][0]) and torch.equal(b, want[i][1]), (rep, i)
    errors = []

    def worker(i):
        try:
            with torch.cuda.stream(streams[i]):
                for _ in range(8):
                    e, b = compute(*cases[i], plans[i])
                    streams[i].synchronize()
                    assert torch.equal(e, want[i][0]) and torch.equal(b, want[i][1]), i
        except Exception as ex:   # noqa: BLE001
            errors.append(ex)

    ts = [threading.Thread(target=worker, args=(i,)) for i in range(len(cases))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_capture_pins_its_buffer_and_failures_give_theirs_back():
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator
    N, n, dt = 32, 3, torch.float32
    plan = plan_of(N, dt, n)
    f, V = inputs(N, n, dt, 9)
    want = compute(N, n, dt, 9, plan)[1]
    op = Operator(Grid3D(N, 8.0), dt, 4)
    op.set_potential(V)
    op.set_exchange(plan, f)
    out = torch.empty_like(f)
    graph = op.block_graph(out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    other = Operator(Grid3D(N, 8.0), dt, 4)   # no plan: the call fails after its first launches
    with pytest.raises(ValueError):
        other.energy_terms(None)
    del other
    for seed in (10, 11):
        compute(N, n, dt, seed, plan)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
