"""GPU: a fused rule whose parameters live on the device, captured into a
CUDA graph after one ordinary call."""
import pytest
import torch

import torchquad_gb300 as tq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm_up", [0, 1, 2])
@pytest.mark.parametrize("method", ["grid", "mc"])
def test_capture_after_warm_up(method, warm_up, cuda):
    dom = torch.tensor([[0.0, 1.0], [0.2, 1.1]], dtype=torch.float64, device=cuda)
    a = torch.tensor([0.4, -0.9], dtype=torch.float64, device=cuda)
    f = tq.ExpSum(2, a=a, c=torch.tensor(1.3, dtype=torch.float64, device=cuda))
    rule, mc = tq.Simpson(), tq.MonteCarlo()

    def call(f):
        if method == "grid":
            return rule.integrate(f, 2, N=21**2, integration_domain=dom)
        return mc.integrate(f, 2, N=1000, integration_domain=dom, seed=5)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(tq.ExpSum(2, a=[0.4, -0.9], c=1.3))  # workspaces and the domain's check, other parameters
        for _ in range(warm_up):
            call(f)
    side.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = call(f)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert out.item() == call(tq.ExpSum(2, a=[0.4, -0.9], c=1.3)).item()
