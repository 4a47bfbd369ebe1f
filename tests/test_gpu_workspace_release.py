"""Kept workspace goes back to the device when asked for and when one of the library's own allocations fails.
The workspace at hand is ten FP32 fields of 128^3, 84 MB; half of that tells it from other tests' leftovers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
KEPT = 10 * 4 * 128 ** 3


def keep():
    """Leaves one block apply's workspace behind and returns the free memory then."""
    from gato_gb300.scf import release_workspace
    from test_gpu_kept_workspace import inputs, plan_of
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator
    release_workspace()
    N, n = 128, 4
    plan = plan_of(N, torch.float32, n)
    f, V = inputs(N, n, torch.float32, 5)
    op = Operator(Grid3D(N, 32.0), torch.float32, 4)
    op.set_potential(V)
    op.set_exchange(plan, f)
    op.apply_block()
    torch.cuda.synchronize()
    del op
    return torch.cuda.mem_get_info()[0], plan   # the plan's memory stays where it is


def test_release_on_request():
    from gato_gb300.scf import release_workspace
    free, plan = keep()
    release_workspace()
    assert torch.cuda.mem_get_info()[0] - free > KEPT // 2
    del plan


def test_release_on_a_failed_allocation():
    from gato_gb300.solvers.poisson import PoissonPlan
    free, plan = keep()
    with pytest.raises(Exception):   # its kernel spectrum alone would take a terabyte
        PoissonPlan(2000, 0.1, 0.05, torch.float64, 1)
    assert torch.cuda.mem_get_info()[0] - free > KEPT // 2
    del plan
