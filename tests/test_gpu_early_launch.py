"""Kernels of a decode step that may start before the kernel in front is complete give what they give one at a time."""
import pytest
import torch

from cpp_minilamma_b200.csrc import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 4, 5])
def test_a_chain_of_products_and_norms(rows):
    """Twelve rounds of wide product, narrow product and norm, each reading what the one before has just written: captured, eager,
    and with a wait behind every kernel."""
    dev, dtype = torch.device("cuda:0"), torch.bfloat16
    g = torch.Generator(device=dev).manual_seed(rows)
    width, inter = 512, 2048
    up = (torch.randn((inter, width), generator=g, device=dev) / width ** 0.5).to(dtype)
    down = (torch.randn((width, inter), generator=g, device=dev) / inter ** 0.5).to(dtype)
    weight = 1.0 + 0.1 * torch.randn(width, generator=g, device=dev)
    first = torch.randn((rows, width), generator=g, device=dev)
    x, h = torch.empty_like(first), torch.empty((rows, width), device=dev, dtype=dtype)
    mid, out = torch.empty((rows, inter), device=dev, dtype=dtype), torch.empty((rows, width), device=dev, dtype=dtype)

    def run(wait):
        x.copy_(first)
        K.add_rmsnorm(x, None, weight, h, 1e-5)
        for _ in range(12):
            for step in (lambda: K.linear_small(h, up, None, mid), lambda: K.linear_small(mid, down, None, out), lambda: K.add_rmsnorm(x, out, weight, h, 1e-5)):
                step()
                if wait:
                    torch.cuda.synchronize()
        return x.clone(), h.clone()

    want = run(True)
    for got in (run(False), run(False)):
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run(False)
    for _ in range(5):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
