"""A plan without strands keeps the transforms of every call on the caller's stream and returns the same bits:
its exchange, captured into a graph, is a chain, and a block graph captured without strands has fewer branches."""
import threading

import pytest
import torch

from test_gpu_in_order import captured_edges
from test_gpu_kept_workspace import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,N,n", [(torch.float64, 20, 3), (torch.float64, 32, 5), (torch.float32, 48, 6),
                                        (torch.float32, 64, 4), (torch.float32, 64, 6), (torch.float32, 70, 5),
                                        (torch.float32, 80, 8), (torch.float32, 98, 7), (torch.float32, 112, 4)])
def test_same_bits_in_one_strand(dtype, N, n):
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    orb, psi = inputs(N, n, dtype, N + n)
    plan = PoissonPlan(N, 0.25, 0.125, dtype, min(pair_fields(n), 6))
    op = Operator(Grid3D(N, 0.25 * N), dtype, 4)
    op.set_potential(psi)
    op.set_exchange(plan, orb)

    def results():
        return [plan.exchange_into(psi, orb, torch.zeros_like(psi)), op.apply(psi), op.apply_block(),
                op.energy_terms(psi), plan.potential(psi), plan.energy(psi)]
    want = results()
    plan.strands(False)
    for a, b in zip(results(), want):
        assert torch.equal(a, b)
    out = torch.zeros_like(psi)
    nodes, edges, widest = captured_edges(lambda: plan.exchange_into(psi, orb, out))
    assert nodes > 2 and edges == nodes - 1 and widest == 1
    torch.cuda.synchronize()


def test_block_graph_and_thread_setting():
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan, get_plan, thread_strands
    N, n = 64, 4
    orb, psi = inputs(N, n, torch.float32, 3)
    plan = PoissonPlan(N, 0.25, 0.125, torch.float32, pair_fields(n))
    op = Operator(Grid3D(N, 0.25 * N), torch.float32, 4)
    op.set_potential(psi)
    op.set_exchange(plan, orb)
    want, out = op.apply_block(), torch.empty_like(orb)
    for strands in (None, False, True):
        graph = op.block_graph(out, strands=strands)
        assert plan.two_strands
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want), strands
    made = []

    def worker():
        thread_strands(False)
        made.append(get_plan(N, 0.25, 0.125, torch.float32).two_strands)
        thread_strands(True)
        made.append(get_plan(N, 0.5, 0.25, torch.float32).two_strands)
    t = threading.Thread(target=worker)
    t.start()
    t.join()
    assert made == [False, True]
    assert get_plan(N, 0.25, 0.125, torch.float32).two_strands
