"""Exchange whose transforms run as two strands on two streams: every mix of full fields, lone fields and
rounds through the buffers against the generic engine, and calls back to back without synchronisation or
replayed from a graph against the same calls one at a time.

Both engines compute the same sums: 25 levels of three axes there and back, a factor of four for their
accumulation, gives 100 eps. The back-to-back and replayed calls run the same kernels on the same inputs,
so they agree exactly.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 100 * 2.0 ** -53, torch.float32: 100 * 2.0 ** -24}
CASES = [(torch.float64, 16), (torch.float64, 50), (torch.float32, 16), (torch.float32, 48), (torch.float32, 64), (torch.float32, 100)]


def inputs(n, N, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    f = torch.rand(n, N, N, N, generator=g, dtype=torch.float64) + 0.1
    return f.to(dtype).cuda(), torch.rand(N, N, N, generator=g, dtype=torch.float64).to(dtype).cuda()


@pytest.mark.parametrize("dtype,N", CASES)
@pytest.mark.parametrize("n,fields", [(2, 1), (3, 2), (4, 2), (5, 3), (5, 2), (6, 3), (7, 1)])
def test_mixes_of_fields(dtype, N, n, fields):
    from gato_gb300.autotune import set_plan
    from gato_gb300.solvers.poisson import PoissonPlan
    plan = PoissonPlan(N, 10.0 / N, 5.0 / N, dtype, fields)
    orb, psi = inputs(n, N, dtype, 10 * N + n)
    got = plan.exchange_into(psi, orb, torch.zeros_like(psi)).double()
    set_plan(plan, 0, 1)
    ref = plan.exchange_into(psi, orb, torch.zeros_like(psi)).double()
    assert float((got - ref).norm() / ref.norm()) < TOL[dtype]


@pytest.mark.parametrize("dtype,N", CASES)
def test_back_to_back_and_replayed(dtype, N):
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    n = 3
    plan = PoissonPlan(N, 10.0 / N, 5.0 / N, dtype, pair_fields(n))
    sets = [inputs(n, N, dtype, k) for k in range(3)]
    ops = []
    for orb, psi in sets:
        op = Operator(Grid3D(N, 10.0), dtype, 4)
        op.set_potential(psi)
        op.set_exchange(plan, orb)
        ops.append(op)

    def calls(k, out):
        ops[k].apply(sets[k][1], out[0])
        ops[k].apply_block(out[1])
        out[2].copy_(ops[k].energy_terms(sets[k][1]))

    def buffers():
        return [torch.zeros_like(sets[0][1]), torch.zeros_like(sets[0][0]),
                torch.zeros(4 + 1, dtype=torch.float64, device="cuda")]
    want = [buffers() for _ in sets]
    for k in range(3):
        calls(k, want[k])
        torch.cuda.synchronize()
    for _ in range(5):
        got = [buffers() for _ in sets]
        for k in (2, 0, 1):
            calls(k, got[k])
        for k in range(3):
            assert all(torch.equal(a, b) for a, b in zip(got[k], want[k])), k
    graph, out = torch.cuda.CUDAGraph(), buffers()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ops[0].apply(sets[0][1], out[0])
        ops[0].apply_block(out[1])
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        ops[0].apply(sets[0][1], out[0])
        ops[0].apply_block(out[1])
    for _ in range(3):
        out[0].zero_(), out[1].zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want[0][0]) and torch.equal(out[1], want[0][1])
