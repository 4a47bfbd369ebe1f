"""An operator without overlap keeps every launch of every call on the caller's stream, in order, and returns
the same bits: a call captured into a graph is a chain, each node after the one before."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def captured_edges(call):
    """(nodes, edges, most edges out of or into a node) of the graph that call() makes of the current stream."""
    cu = C.CDLL("libcuda.so.1")
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph, n, e = C.c_void_p(), C.c_size_t(), C.c_size_t()
    with torch.cuda.stream(stream):
        call()   # the stream's scratch is allocated here
        stream.synchronize()
        assert cu.cuStreamBeginCapture_v2(C.c_void_p(stream.cuda_stream), 2) == 0   # relaxed
        try:
            call()
        finally:
            assert cu.cuStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(graph)) == 0
    try:
        assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
        assert cu.cuGraphGetEdges_v2(graph, None, None, None, C.byref(e)) == 0
        src, dst = (C.c_void_p * e.value)(), (C.c_void_p * e.value)()
        data = (C.c_uint64 * e.value)()   # eight bytes an edge
        assert cu.cuGraphGetEdges_v2(graph, src, dst, data, C.byref(e)) == 0
        return n.value, e.value, max(list(q).count(x) for q in (src, dst) for x in q)
    finally:
        cu.cuGraphDestroy(graph)


@pytest.mark.parametrize("dtype,N", [(torch.float64, 32), (torch.float32, 64)])
def test_in_order(dtype, N):
    from gato_gb300 import _lib
    from gato_gb300.grid import Grid3D
    from gato_gb300.scf import Operator, pair_fields
    from gato_gb300.solvers.poisson import PoissonPlan
    n = 3
    gen = torch.Generator(device="cuda").manual_seed(N)
    f = torch.rand(n, N, N, N, generator=gen, dtype=torch.float64, device="cuda").to(dtype)
    V = torch.rand(N, N, N, generator=gen, dtype=torch.float64, device="cuda").to(dtype)
    op = Operator(Grid3D(N, 0.25 * N), dtype, 4)
    op.set_potential(V)
    op.set_exchange(PoissonPlan(N, 0.25, 0.125, dtype, pair_fields(n)), f)
    out = [torch.empty_like(V), torch.empty_like(f), torch.empty(5, dtype=torch.float64, device="cuda")]
    P = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    calls = [lambda: op.apply(V, out[0]), lambda: op.apply_block(out[1]),
             lambda: _lib.call("gato_op_energy_terms", op.handle, P(V), P(out[2]), C.c_void_p(_lib.stream()))]
    results = []
    for on in (True, False):
        op.overlap(on)
        for t, call in zip(out, calls):
            t.zero_()
            call()
        results.append([t.clone() for t in out])
    for a, b in zip(*results):
        assert torch.equal(a, b)
    for call in calls:
        nodes, edges, widest = captured_edges(call)
        assert nodes > 2 and edges == nodes - 1 and widest == 1
    torch.cuda.synchronize()
