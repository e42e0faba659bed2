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


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("n", [700, 30000])
def test_captured_row_orders(n, precision, cuda):
    """A Deconvolution and the gradients of a Convolution whose row orders are made while they are recorded: every replay makes
    them again, the children's tiles from cursors that the replay before has left as it found them."""
    import sparseconvnet_b200 as scn
    from sparseconvnet_b200 import SCN
    torch.manual_seed(n)
    planes, pts = 160, _surface(n, 96)
    up = scn.Deconvolution(3, planes, planes, 2, 2, True).to(cuda).requires_grad_(False)
    first = scn.Convolution(3, 4, 4, 2, 2, False).to(cuda).requires_grad_(False)
    w = torch.randn(8, 1, planes, planes, device=cuda)
    size, half, two = torch.LongTensor([96] * 3), torch.LongTensor([48] * 3), torch.LongTensor([2] * 3)

    def start():
        x = scn.InputLayer(3, 96, mode=4)([pts, torch.randn(n, 4, device=cuda)])
        return x.metadata, first(x).features.size(0), x.features.size(0)

    def run(m, coarse, fine, d_in, dw):
        y = up(scn.SparseConvNetTensor(coarse, m, half)).features
        SCN.Convolution_backward(size, half, two, two, m, fine, d_in, coarse, w, dw, None)
        return y
    try:
        scn.set_precision(precision)
        scn.set_backward_precision(precision)
        m, n_coarse, n_fine = start()
        coarse, fine = torch.randn(n_coarse, planes, device=cuda), torch.randn(n_fine, planes, device=cuda)
        d_in, dw = torch.empty_like(fine), torch.empty_like(w)
        run(start()[0], coarse, fine, d_in, dw)  # (what the process sets up once)
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            y = run(m, coarse, fine, d_in, dw)
        for _ in range(3):
            coarse.copy_(torch.randn_like(coarse))
            fine.copy_(torch.randn_like(fine))
            for t in (y, d_in, dw):
                t.fill_(float("nan"))
            graph.replay()
            torch.cuda.synchronize()
            other = torch.empty_like(d_in), torch.empty_like(dw)
            want = run(start()[0], coarse, fine, *other)
            for a, b in ((y, want), (d_in, other[0]), (dw, other[1])):
                assert torch.equal(a, b)
        m.poll_errors()
        del m
        del graph
    finally:
        scn.set_precision("fp32")
        scn.set_backward_precision("fp32")


def _used():
    import ctypes as C
    from sparseconvnet_b200._lib import check, lib
    reserved, used = C.c_uint64(), C.c_uint64()
    check(lib.scn_memory_usage(C.byref(reserved), C.byref(used)))
    return reserved.value, used.value


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("n,coords", [(3000, "cpu"), (3000, "cuda"), (300, "cpu")])
def test_nothing_is_lost_when_memory_runs_out(n, coords, precision, cuda):
    """Input layer, rulebooks, row order, forward and backward pass with the first, second, ... allocation failing: an error
    each time -- or, where a layer does with less, the same results to rounding --, every block given back with the object, and the
    next pass gives what an undisturbed one does."""
    import sparseconvnet_b200 as scn
    from sparseconvnet_b200 import SCN
    from sparseconvnet_b200._lib import ScnError, lib
    torch.manual_seed(n)
    pts = _surface(n, 48).to(coords)
    feats = torch.randn(n, 32, device=cuda)
    size, half, three, two = torch.LongTensor([48] * 3), torch.LongTensor([24] * 3), torch.LongTensor([3] * 3), torch.LongTensor([2] * 3)
    w = [torch.randn(27, 1, 32, 64, device=cuda), torch.randn(8, 1, 64, 40, device=cuda)]
    none = torch.empty(0)
    pending = [0]

    def run():
        m = SCN.Metadata_3()
        try:
            x = SCN.InputLayer_updateOutput(m, size, pts, feats, None, 0, 3)
            y, z = (feats.new_empty(0) for _ in range(2))
            SCN.SubmanifoldConvolution_updateOutput(size, three, m, x, y, w[0], none)
            SCN.Convolution_updateOutput(size, half, two, two, m, y, z, w[1], none)
            g = [torch.empty_like(t) for t in (w[0], w[1], x, y)]
            SCN.Convolution_backward(size, half, two, two, m, y, g[3], torch.ones_like(z), w[1], g[1], None)
            SCN.SubmanifoldConvolution_backward(size, three, m, x, g[2], g[3], w[0], g[0], None)
            mean, var, d_b = (torch.empty(64, device=cuda) for _ in range(3))
            out, d_in = torch.empty_like(y), torch.empty_like(y)
            SCN.BatchNormalization_updateOutput(y, out, mean, var, torch.zeros(64, device=cuda), torch.ones(64, device=cuda),
                                                none, none, 1e-4, 0.9, True, 0.0)
            SCN.BatchNormalization_backward(y, d_in, out, g[3], mean, var, None, None, none, none, None, d_b, 0.0)
            return [x, y, z] + g
        finally:
            pending[0] = lib.scn_test_fail_allocation(0)
            del m

    try:
        scn.set_precision(precision)
        scn.set_backward_precision(precision)
        want = run()
        torch.cuda.synchronize()
        before = _used()[1]
        failed = 0
        for which in range(1, 200):
            lib.scn_test_fail_allocation(which)
            try:
                got = run()
                if pending[0]:  # there was no such allocation any more
                    break
                # (sums of at most 27 x 64 fp32 products, and of 3000 of them in the weights' gradients)
                assert precision == "fp32" and all(float((a - b).norm()) <= 1e-5 * float(b.norm()) for a, b in zip(got, want)), which
            except ScnError as e:
                assert "out of memory" in str(e), e
                failed += 1
            assert _used()[1] == before, (which, _used()[1] - before)
        assert failed > 15 and which > failed
        assert all(torch.equal(a, b) for a, b in zip(run(), want))
        assert _used()[1] == before
    finally:
        scn.set_precision("fp32")
        scn.set_backward_precision("fp32")


def test_weight_gradient_scratch_is_bounded(cuda):
    """125 offsets of 256 x 256 weights are 33 MB per chunk of tiles: 25 chunks of 48 tiles, of which at most 256 MB at a
    time; the gradient is the sum of all of them."""
    import sparseconvnet_b200 as scn
    from sparseconvnet_b200 import SCN
    from sparseconvnet_b200._lib import check, lib
    torch.manual_seed(3)
    n, planes = 150000, 256
    cell = torch.randperm(96 ** 3, device=cuda)[:n]
    pts = torch.stack([cell // 96 ** 2, cell // 96 % 96, cell % 96], 1)
    x = scn.InputLayer(3, 96, mode=0)([pts, torch.zeros(n, 1, device=cuda)])
    w, dw = torch.randn(125, 1, planes, planes, device=cuda), torch.empty(125, 1, planes, planes, device=cuda)
    f, g = torch.randn(n, planes, device=cuda), torch.randn(n, planes, device=cuda)
    five = torch.LongTensor([5] * 3)

    def backward(f, g, w, dw):
        SCN.SubmanifoldConvolution_backward(x.spatial_size, five, x.metadata, f, None, g, w, dw, None)
    backward(f[:, :64].contiguous(), g[:, :64].contiguous(), w[:, :, :64, :64].contiguous(),
             torch.empty(125, 1, 64, 64, device=cuda))  # the rulebook and its row order
    torch.cuda.synchronize()
    check(lib.scn_trim_memory(0))
    before = _used()[0]
    backward(f, g, w, dw)
    torch.cuda.synchronize()
    rows = 2 * n * planes * 6      # both sides as three bf16 parts
    assert _used()[0] - before <= 1.25 * (rows + (256 << 20)) + (64 << 20)
    rules = x.metadata.rulebook(0, x.spatial_size, five)
    for k in (0, 31, 62, 124):
        r = rules[k].long()
        want = f[r[:, 0]].double().t() @ g[r[:, 1]].double()
        assert float((dw[k, 0] - want).norm() / want.norm()) <= 1e-5
    x.metadata.poll_errors()


def test_batchnorm_scratch_is_bounded(cuda):
    """Statistics of 4 095 planes on 65 k rows, 1 024 chunks: what a chunk leaves is 16 bytes a plane, 67 MB if each left its own.
    A chunk's fp32 sums are of eight rows at most (eight roundings, and one of a square), and added in double."""
    from sparseconvnet_b200._lib import check, lib
    for n, planes in ((65536, 4095), (65535, 515), (700, 4095), (1, 2049)):
        torch.manual_seed(planes)
        x, sums = torch.randn(n, planes, device=cuda), torch.empty(2 * planes + 1, dtype=torch.float64, device=cuda)
        torch.cuda.synchronize()
        check(lib.scn_trim_memory(0))
        before = _used()[0]
        check(lib.scn_batchnorm_moments(x.data_ptr(), n, planes, planes, sums.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert _used()[0] - before <= 40 << 20
        for got, power in ((sums[:planes], 1), (sums[planes:2 * planes], 2)):
            want, scale = (torch.zeros(planes, dtype=torch.float64, device=cuda) for _ in range(2))
            for part in x.split(8192):
                want += (part.double() ** power).sum(0)
                scale += (part.double() ** power).abs().sum(0)
            assert bool(((got - want).abs() <= 9 * 2.0 ** -24 * scale).all())
