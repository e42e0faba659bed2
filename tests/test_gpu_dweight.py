"""Weight gradients of the convolutions (k_conv_dweight_mma, k_dweight_tile) against a float64 product over the exported rulebook.

Multiples of 32 planes, more than 32 on one side, run on k_dweight_tile from 2048 rows, with blocks of 32 or 64 planes per side;
its six bf16 products drop 2^-24 of a product and its running sums lose at most 2^-24 per instruction: 384 of them in the sums
of the large parts, 1 152 in those of the others, which are 2^-8 as large.

Tolerance: three tf32 products of the hi / lo split drop lo x lo and a bit of lo, 2^-22 of a product, and n fp32
additions of random sign add 2^-24 sqrt(n) of the running sum: below 1e-5 of the largest entry for the row counts here;
1e-4 is the fp32 bar of the package."""
import numpy as np
import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout", [(1, 8), (3, 32), (8, 16), (24, 20), (32, 33), (31, 64), (64, 96), (96, 64), (96, 96),
                                      (100, 160), (192, 96), (33, 1), (32, 64), (64, 32), (40, 36), (12, 68)])
@pytest.mark.parametrize("n,size", [(40, 12), (6000, 40), (30001, 96)])
def test_weight_gradient(n, size, cin, cout, cuda):
    _weight_gradient(n, size, cin, cout, cuda, True)


def _weight_gradient(n, size, cin, cout, cuda, transposed):
    """The gradients of three layers (two: without the transposed one), and that the kernel meant for the shape ran."""
    import sparseconvnet_b200 as scn
    rng = np.random.default_rng(n + cin)
    pts = rng.integers(0, size, (n, 3))
    pts[:, 2] = size // 2 + size // 5 * np.sin(pts[:, 0] / 6.0) + rng.integers(0, 2, n)
    x = scn.InputLayer(3, size, mode=4)([torch.from_numpy(pts), torch.zeros(n, 1, device=cuda)])
    up_size = torch.LongTensor([size // 2] * 3)
    torch.manual_seed(cin)
    for layer in (scn.SubmanifoldConvolution(3, cin, cout, 3, True), scn.Convolution(3, cin, cout, 2, 2, False),
                  scn.Deconvolution(3, cin, cout, 2, 2, False)):
        layer.to(cuda)
        md, filt = x.metadata, [2, 2, 2]
        if isinstance(layer, scn.Deconvolution):
            if not transposed:
                continue
            rows, spatial = md.getNActive(up_size), up_size
        else:
            rows, spatial = x.features.size(0), x.spatial_size
        f = torch.randn(rows, cin, device=cuda, requires_grad=True)
        y = layer(scn.SparseConvNetTensor(f, md, spatial))
        g = torch.randn_like(y.features)
        y.features.backward(g)
        torch.cuda.synchronize()
        table = x.features.size(0) if isinstance(layer, scn.SubmanifoldConvolution) else md.getNActive(up_size)
        tile = table >= 2048 and cin % 32 == 0 and cout % 32 == 0 and max(cin, cout) > 32
        thin = cin <= 3 and cout <= 32 and not isinstance(layer, scn.Deconvolution)
        assert scn.SCN.lib.scn_last_dweight_kernel() == (2 if tile else 3 if thin else 1)
        if isinstance(layer, scn.SubmanifoldConvolution):
            rules = md.rulebook(0, x.spatial_size, [3, 3, 3])
        else:
            rules = md.rulebook(1, x.spatial_size, filt, filt)
        if isinstance(layer, scn.Deconvolution):
            rules = [r.flip(1) for r in rules]
        fd, gd = f.detach().double(), g.double()
        want = torch.stack([fd[r[:, 0].long()].t() @ gd[r[:, 1].long()] for r in rules])
        e = helpers.rel_err(layer.weight.grad[:, 0].double().cpu().numpy(), want.cpu().numpy())
        assert e <= helpers.FP32_TOL, (layer, e)
        want = torch.zeros(rows, cin, dtype=torch.float64, device=cuda)
        for r, w in zip(rules, layer.weight.detach().double()[:, 0]):
            want.index_add_(0, r[:, 0].long(), gd[r[:, 1].long()] @ w.t())
        e = helpers.rel_err(f.grad.double().cpu().numpy(), want.cpu().numpy())
        assert e <= helpers.FP32_TOL, (layer, "input gradient", e)


@pytest.mark.parametrize("cin,cout", [(1, 1), (4, 32), (32, 20), (33, 40), (48, 20), (100, 7)])
@pytest.mark.parametrize("n", [1, 31, 512, 513, 70001])
def test_network_in_network_gradients(n, cin, cout, cuda):
    """One fp32 sum of n products per weight, in chunks of at least 512 rows: 2^-24 sqrt(n) of the largest, far below the
    package's fp32 bar."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(n + cin)
    layer = scn.NetworkInNetwork(cin, cout, True).to(cuda)
    f = torch.randn(n, cin, device=cuda, requires_grad=True)
    y = layer(scn.SparseConvNetTensor(f, None, None)).features
    g = torch.randn_like(y)
    y.backward(g)
    fd, gd, wd = f.detach().double(), g.double(), layer.weight.detach().double()
    for got, want in ((y, fd @ wd + layer.bias.detach().double()), (f.grad, gd @ wd.t()), (layer.weight.grad, fd.t() @ gd),
                      (layer.bias.grad, gd.sum(0))):
        assert helpers.rel_err(got.detach().double().cpu().numpy(), want.cpu().numpy()) <= helpers.FP32_TOL


@pytest.mark.parametrize("planes", [4, 20, 32, 36, 100])
@pytest.mark.parametrize("n", [5, 33, 64, 257, 40001])
def test_batchnorm_training_sums(n, planes, cuda):
    """k_bn_stats4 and k_bn_back_sums4 against torch in float64; fp32 sums of a few hundred values each, added in double.
    At least five rows: the gradient is g minus its projections on 1 and on the normalised row, and with two rows nothing
    but eps / var of it is left, rounding errors of 2^-23 g times up to var / eps = 1e4."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(n + planes)
    layer = scn.BatchNormLeakyReLU(planes, leakiness=0.25).to(cuda)
    torch.nn.init.uniform_(layer.weight, 0.5, 1.5)
    torch.nn.init.uniform_(layer.bias, -1, 1)
    x = torch.randn(n, planes, device=cuda, requires_grad=True)
    y = layer(scn.SparseConvNetTensor(x, None, None)).features
    g = torch.randn_like(y)
    y.backward(g)
    xd, w, b = (t.detach().double().requires_grad_() for t in (x, layer.weight, layer.bias))
    mean, var = xd.mean(0), xd.var(0, unbiased=False)
    z = (xd - mean) / torch.sqrt(var + layer.eps) * w + b
    yd = torch.where(z > 0, z, 0.25 * z)
    yd.backward(torch.where((y.detach() > 0) == (z.detach() > 0), g, torch.zeros_like(g)).double())
    assert helpers.rel_err(y.detach().double().cpu().numpy(), yd.detach().cpu().numpy()) <= helpers.FP32_TOL
    same = ((y.detach() > 0) == (z.detach() > 0)).all()
    if same:  # (a value within rounding of zero may take the other slope)
        for got, want in ((x.grad, xd.grad), (layer.weight.grad, w.grad), (layer.bias.grad, b.grad)):
            assert helpers.rel_err(got.double().cpu().numpy(), want.cpu().numpy()) <= helpers.FP32_TOL


@pytest.mark.parametrize("tiles,extra", [(148, 0), (148, 1), (149, 0), (4096, 0), (4096, 1), (65535, 0), (65535, 1)])
def test_tiles_by_work(tiles, extra, cuda):
    """Row counts around the levels whose tiles are sorted by their offsets (149 to 65535 tiles of 128 rows; up to 4096 of
    them the sort keeps its bins in registers), masks of every fill: outputs and weight gradient, each tile once."""
    import sparseconvnet_b200 as scn
    n = tiles * 128 + extra
    size = int(np.ceil((2.3 * n) ** (1 / 3)))
    torch.manual_seed(tiles + extra)
    cell = (torch.rand(size ** 3, device=cuda) < torch.arange(size ** 3, device=cuda) / size ** 3).nonzero()[:, 0]
    cell = cell[torch.randperm(len(cell), device=cuda)[:n]]
    pts = torch.stack([cell // size ** 2, cell // size % size, cell % size], 1)
    assert len(pts) == n
    x = scn.InputLayer(3, size, mode=0)([pts.cpu(), torch.randn(n, 16, device=cuda)])
    layer = scn.SubmanifoldConvolution(3, 16, 40, 3, False).to(cuda)
    f = x.features
    g = torch.randn_like(layer(x).features)
    rules = [r.long() for r in x.metadata.rulebook(0, x.spatial_size, [3, 3, 3])]
    w = layer.weight.detach()[:, 0]
    want = torch.zeros(n, 40, dtype=torch.float64, device=cuda)
    for r, wk in zip(rules, w.double()):
        want.index_add_(0, r[:, 1], f.double()[r[:, 0]] @ wk)
    want_w = torch.stack([f[r[:, 0]].double().t() @ g[r[:, 1]].double() for r in rules])
    try:
        for precision in ("fp32", "tf32x3"):
            scn.set_precision(precision)
            layer.weight.grad = None
            y = layer(x).features
            y.backward(g)
            assert float((y.detach() - want).abs().max() / want.abs().max()) <= helpers.FP32_TOL, precision
            e = float((layer.weight.grad[:, 0] - want_w).abs().max() / want_w.abs().max())
            assert e <= helpers.FP32_TOL, (precision, e)
        x.metadata.poll_errors()
    finally:
        scn.set_precision("fp32")


@pytest.mark.parametrize("cin", [1, 2, 3])
@pytest.mark.parametrize("cout", [1, 20, 32])
@pytest.mark.parametrize("n,size", [(1, 8), (300, 16), (6000, 40), (120001, 160)])
def test_thin_weight_gradient(n, size, cin, cout, cuda):
    """k_conv_dweight_thin: batches of 32 rows, nine offsets and the planes with and without remainders."""
    _weight_gradient(n, size, cin, cout, cuda, False)


@pytest.mark.parametrize("cin,cout", [(8, 16), (24, 24), (32, 32), (48, 48), (80, 36), (100, 160), (64, 64), (64, 96)])
@pytest.mark.parametrize("n,size", [(6000, 40), (60000, 120)])
def test_weight_gradient_is_as_accurate_as_fp32_sums(n, size, cin, cout, cuda):
    """Products of one sign, where everything that is cut off instead of rounded adds up.  Rounded to nearest, the two tf32
    parts of an operand leave out at most 2^-23 of it and lo x lo 2^-22 of a product, of either sign, and n fp32 additions
    2^-24 sqrt(n) / 2 of the sum: below 5e-7 for the 3 k rules of an entry and chunk here.  (Parts cut off: 4e-6 to 8e-6.)
    On k_dweight_tile (multiples of 32 planes, more than 32 on a side) up to 384 instructions each cut 2^-24 of a running sum
    that is half of the last one on average: 1.2e-5."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(cin)
    pts = torch.randint(0, size, (n, 3))
    pts[:, 2] = size // 2 + (size // 5 * torch.sin(pts[:, 0] / 6.0)).long() + torch.randint(0, 2, (n,))
    x = scn.InputLayer(3, size, mode=4)([pts, torch.zeros(n, 1, device=cuda)])
    layer = scn.SubmanifoldConvolution(3, cin, cout, 3, False).to(cuda)
    f = torch.rand(x.features.size(0), cin, device=cuda)
    y = layer(scn.SparseConvNetTensor(f, x.metadata, x.spatial_size)).features
    g = torch.rand_like(y)
    y.backward(g)
    want = torch.stack([f[r[:, 0].long()].double().t() @ g[r[:, 1].long()].double()
                        for r in x.metadata.rulebook(0, x.spatial_size, [3, 3, 3])])
    e = float((layer.weight.grad[:, 0] - want).norm() / want.norm())
    assert e <= (1.2e-5 if cin % 32 == 0 and cout > 32 and cout % 32 == 0 else 5e-7), e


def _affine(features, weight, bias):
    """NetworkInNetwork's training path on these operands."""
    from sparseconvnet_b200 import autograd
    return autograd.rows_affine(features, weight, bias)


def test_network_in_network_takes_what_a_matrix_product_takes(cuda):
    """Operands that torch's product accepts or refuses, on the training path: a transposed weight, offset, strided and
    double-precision features, a bias of one value, one of a wrong length, operands on the host."""
    torch.manual_seed(0)
    flat = torch.randn(1 + 600 * 32, device=cuda)
    base = torch.randn(20, 32, device=cuda).t()
    for f in (flat[1:].view(600, 32), flat[:600 * 32].view(32, 600).t(), flat[:600 * 32].view(600, 32).double()):
        for bias in (None, torch.randn(1, device=cuda, dtype=f.dtype), torch.randn(20, device=cuda, dtype=f.dtype)):
            w = base.to(f.dtype).detach().requires_grad_()
            got = _affine(f, w, bias)
            want = f.double() @ w.detach().double() + (bias.double() if bias is not None else 0)
            assert got.dtype == f.dtype and float((got.detach() - want).abs().max()) < 1e-4
            got.sum().backward()
            assert float((w.grad - f.double().sum(0)[:, None]).abs().max()) < 1e-2
    f, w = flat[:-1].view(600, 32), torch.randn(32, 20, device=cuda, requires_grad=True)
    g = torch.randn(1 + 600 * 20, device=cuda)[1:].view(600, 20)   # an offset gradient
    fr = f.clone().requires_grad_()
    _affine(fr, w, None).backward(g)
    assert float((fr.grad.double() - g.double() @ w.detach().double().t()).abs().max()) < 1e-4
    for bad in ((f, w, torch.zeros(19, device=cuda)), (f, w, torch.zeros(20)), (f, w.detach().cpu().requires_grad_(), None),
                (f, torch.randn(31, 20, device=cuda, requires_grad=True), None)):
        with pytest.raises(RuntimeError):
            _affine(*bad)


def test_network_in_network_under_torchs_transforms(cuda):
    """Second derivatives, forward mode, vmap, torch.func.grad, autocast and saved-tensor hooks see a matrix product."""
    import torch.autograd.forward_ad as fwd
    torch.manual_seed(1)
    f = torch.randn(50, 12, device=cuda)
    w, b = torch.randn(12, 8, device=cuda, requires_grad=True), torch.randn(8, device=cuda, requires_grad=True)

    def plain(f, w, b):
        return f @ w + b

    for view in (lambda t: t, lambda t: t.t().contiguous().t()):   # contiguous and strided rows
        second = []
        for op in (_affine, plain):
            x = f.clone().requires_grad_()
            y = op(view(x * x), w, b)
            (gx,) = torch.autograd.grad((y ** 3).sum(), x, create_graph=True)
            second.append(torch.autograd.grad((gx ** 2).sum(), (x, w)))
        assert all(torch.allclose(p, q, rtol=1e-3, atol=1e-2 * float(q.abs().max())) for p, q in zip(*second))
    with fwd.dual_level():
        t = torch.randn_like(f)
        out = fwd.unpack_dual(_affine(fwd.make_dual(f, t), w, b))
        assert out.tangent is not None and torch.allclose(out.tangent, t @ w, atol=1e-4)
    grad = torch.func.grad(lambda f: _affine(f, w, b).pow(2).sum())(f)
    assert torch.allclose(grad, 2 * plain(f, w, b) @ w.t(), atol=1e-3)
    batched = torch.func.vmap(lambda f: _affine(f, w, b))(torch.stack([f, 2 * f]))
    assert torch.allclose(batched[1], plain(2 * f, w, b), atol=1e-4)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert _affine(f, w, None).dtype == (f @ w).dtype
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t) or t, lambda t: t):
        _affine(f.clone().requires_grad_(), w, b)
    assert len(seen) == 2
