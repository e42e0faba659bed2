"""The library's memory: under stream capture, after failing calls, and how much of it a call takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _surface(n, size, seed=0):
    g = torch.Generator().manual_seed(seed)
    pts = torch.randint(0, size, (n, 3), generator=g)
    pts[:, 2] = size // 2 + (size // 5 * torch.sin(pts[:, 0] / 6.0)).long() + torch.randint(0, 2, (n,), generator=g)
    return pts


@pytest.mark.parametrize("precision", ["fp32", "tf32x3", "bf16"])
@pytest.mark.parametrize("n", [700, 30000])
def test_captured_convolution(n, precision, cuda):
    """A convolution on a finished rulebook recorded into a CUDA graph: its scratch belongs to the graph, so calls between
    the capture and a replay neither disturb the replay nor are disturbed by it."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(n)
    pts = _surface(n, 96)
    layers = [scn.SubmanifoldConvolution(3, 64, 96, 3, True).to(cuda), scn.Convolution(3, 96, 64, 2, 2, False).to(cuda)]
    try:
        scn.set_precision(precision)
        with torch.no_grad():
            def run(x):
                for layer in layers:
                    x = layer(x)
                return x.features
            x = scn.InputLayer(3, 96, mode=4)([pts, torch.randn(n, 64, device=cuda)])
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                run(x)  # rulebooks, row orders and weight images
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                y = run(x)
            x.features.copy_(torch.randn_like(x.features))
            want = run(x).clone()
            torch.cuda.synchronize()
            for seed in range(3):
                with torch.cuda.stream(side):  # blocks of the sizes the graph was recorded with
                    o = scn.InputLayer(3, 96, mode=4)([_surface(n, 96, seed + 1), torch.ones(n, 64, device=cuda)])
                    got = run(o).clone()
                    graph.replay()
                    again = run(o)
                torch.cuda.synchronize()
                assert torch.equal(y, want)
                assert torch.equal(got, again)
            x.metadata.poll_errors()
            del graph
    finally:
        scn.set_precision("fp32")
