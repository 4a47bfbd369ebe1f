"""Where FP32 calls fork a second strand: by shape and field count (two pair densities a field), on both sides of
each limit, accumulating and to J fields. A second strand shows as more launches in the captured call than the plan
makes without strands; either way the generic engine's results, to 100 eps (25 levels of three axes there and back,
a factor of four for their accumulation)."""
import pytest
import torch

from test_gpu_in_order import captured_edges
from test_gpu_kept_workspace import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n,block,forks", [
    (60, 6, False, False), (64, 4, False, False), (64, 5, False, True), (70, 2, False, False), (70, 3, False, True),
    (80, 4, False, True), (90, 8, False, True), (90, 9, False, False), (98, 4, False, True), (98, 5, False, False),
    (108, 4, False, True), (108, 5, False, False), (144, 4, False, False),
    (60, 4, True, False), (64, 2, True, False), (64, 3, True, True), (72, 4, True, True), (72, 5, True, False),
    (84, 3, True, True), (84, 4, True, False), (112, 4, True, True), (112, 5, True, False), (140, 3, True, False)])
def test_rule(N, n, block, forks):
    from gato_gb300.autotune import set_plan
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    orb, psi = inputs(N, n, torch.float32, N + n)
    plan = PoissonPlan(N, 10.0 / N, 5.0 / N, torch.float32, pair_fields(n) if block else 5)
    op = Operator(Grid3D(N, 10.0), torch.float32, 4)
    op.set_exchange(plan, orb)
    op.tune(1)   # the block apply through J fields
    out = torch.zeros_like(orb if block else psi)

    def call():
        return op.apply_block(out) if block else plan.exchange_into(psi, orb, out)
    nodes = []
    for on in (True, False):
        plan.strands(on)
        nodes.append(captured_edges(call)[0])
    plan.strands(True)
    assert (nodes[0] > nodes[1]) == forks, nodes
    got = (call() if block else plan.exchange_into(psi, orb, torch.zeros_like(psi))).double()
    set_plan(plan, 0, 1)
    op.tune(0)
    ref = (call() if block else plan.exchange_into(psi, orb, torch.zeros_like(psi))).double()
    assert float((got - ref).norm() / ref.norm()) < 100 * 2.0 ** -24
