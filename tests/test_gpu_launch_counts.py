"""The launch counts that the reports give are those of the launches made, counted in a captured graph."""
from __future__ import annotations

import pytest
import torch

from pyocean_b200 import workloads as W
from pyocean_b200.batch import Domain, DomainBatch, batch_launches, sequential_launches, sequential_step
from pyocean_b200.step import ALETracerStep

pytestmark = pytest.mark.gpu


def _kernels(call) -> int:
    from cuda.bindings import runtime as rt
    call(torch.cuda.current_stream().cuda_stream)                 # outside the capture first
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call(torch.cuda.current_stream().cuda_stream)
    err, _, n = rt.cudaGraphGetNodes(graph.raw_cuda_graph())
    err, nodes, n = rt.cudaGraphGetNodes(graph.raw_cuda_graph(), n)
    kinds = [rt.cudaGraphNodeGetType(x)[1] for x in nodes[:n]]
    return sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)


@pytest.mark.parametrize("nt,n,ny,nx", [(1, 20, 8, 9), (2, 20, 200, 200), (3, 5, 400, 400), (2, 75, 40, 40), (3, 75, 388, 389),
                                        (1, 97, 20, 20), (2, 97, 20, 20), (3, 97, 20, 20), (1, 50, 143, 141)])
def test_step(nt, n, ny, nx):
    dev = torch.device("cuda", 0)
    st = ALETracerStep(nt, n, ny, nx, 100.0, 0, 2, device=dev)
    z = lambda *s: torch.ones(s, dtype=torch.float64, device=dev)                        # noqa: E731
    C, V, Qx, Qy, out = z(nt, n, ny, nx), z(n, ny, nx), z(n, ny, nx + 1), z(n, ny + 1, nx), z(nt, n, ny, nx)
    ok, wet = torch.ones((n, ny, nx), dtype=torch.uint8, device=dev), torch.ones((ny, nx), dtype=torch.uint8, device=dev)

    def call(_):
        st.remap(V, st.advect(C, V, V, Qx, Qy, ok), V, wet, out)

    assert _kernels(call) == st.launches_per_step


@pytest.mark.parametrize("nf", [1, 2])
@pytest.mark.parametrize("boxes", [[(20, 20, 5, 1)], [(30, 20, 20, 2), (20, 20, 97, 1)], [(16, 12, 3, 1)] * 65,
                                   [(240, 200, 50, 1)] * 2, [(150, 150, 30, 3), (90, 90, 30, 2)], [(150, 90, 75, 1)] * 3])
def test_batch(boxes, nf):
    dev = torch.device("cuda", 0)
    doms = [Domain.from_workload(W.zstar_box(seed=i, nx=a, ny=b, n=n, nt=nt), dev) for i, (a, b, n, nt) in enumerate(boxes)]
    batch = DomainBatch(doms, remap_nf=nf)
    plan = batch.plan
    assert _kernels(lambda st: plan.step(0, nf, False, st)) == batch.launches_per_step == batch_launches(
        [d.shape for d in doms], nf)
    if len(doms) < 5:
        assert _kernels(lambda st: sequential_step(doms, 0, stream=st)) == sequential_launches(doms)
