"""Layers whose fine rows have one rule each (filter = stride), on tiles made from the parents' side in one launch: against
float64 over the exported rulebook, at the edges of tiles and with offsets that few rows or none have."""
import numpy as np
import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu


def _points(n, dim, size, corner):
    rng = np.random.default_rng(n + dim)
    pts = rng.integers(0, size, (4 * n + 8, dim))
    if corner:  # every site at the same place of its cell: one offset has all rules
        pts = pts // 2 * 2 + 1
    pts = np.unique(pts, axis=0)
    pts = pts[rng.permutation(len(pts))][:n]
    return np.concatenate([pts, rng.integers(0, 2, (len(pts), 1))], axis=1)


# fp32: multiply-adds or three bf16 parts, sums of cin products; the others: what the split leaves out, one bf16 product
@pytest.mark.parametrize("precision,tol", [("fp32", 1e-6), ("tf32x3", helpers.FP32_TOL), ("bf16", helpers.TC_TOL)])
@pytest.mark.parametrize("n,dim,filt,corner", [(1, 3, 2, False), (127, 3, 2, False), (128, 3, 2, True), (129, 3, 2, True),
                                               (5000, 3, 2, False), (40000, 3, 2, False), (3000, 2, 3, False), (9000, 3, 3, False),
                                               (6000, 4, 2, False)])
def test_children(n, dim, filt, corner, precision, tol, cuda):
    import sparseconvnet_b200 as scn
    size = {2: 96, 3: 48, 4: 24}[dim]
    coords = _points(n, dim, size, corner)
    cin, cout = 64, 48
    torch.manual_seed(n)
    up = scn.Deconvolution(dim, cin, cout, filt, filt, True).to(cuda)
    down = scn.Convolution(dim, cout, cin, filt, filt, False).to(cuda)
    up.bias.data.normal_()
    coarse = torch.LongTensor([size // filt] * dim)
    try:
        scn.set_precision(precision)
        scn.set_backward_precision(precision)
        # mode 1: no rows that are in no map
        x = scn.InputLayer(dim, size, mode=1)([torch.from_numpy(coords), torch.zeros(len(coords), 1, device=cuda)])
        fine = torch.randn(x.features.size(0), cout, device=cuda, requires_grad=True)
        y = down(scn.SparseConvNetTensor(fine, x.metadata, x.spatial_size)).features
        g = torch.randn_like(y)
        y.backward(g)
        f = torch.randn(y.size(0), cin, device=cuda)
        with torch.no_grad():
            z = up(scn.SparseConvNetTensor(f, x.metadata, coarse)).features
        x.metadata.poll_errors()
    finally:
        scn.set_precision("fp32")
        scn.set_backward_precision("fp32")
    want = up.bias.detach().double().expand(z.shape).clone()
    grad = torch.zeros(fine.shape, dtype=torch.float64, device=cuda)
    seen = 0
    for r, w, v in zip(x.metadata.rulebook(1, x.spatial_size, [filt] * dim, [filt] * dim), up.weight.detach().double()[:, 0],
                       down.weight.detach().double()[:, 0]):
        r = r.long()
        seen += len(r)
        want.index_add_(0, r[:, 0], f.double()[r[:, 1]] @ w)
        grad.index_add_(0, r[:, 0], g.double()[r[:, 1]] @ v.t())
    assert seen == len(fine)
    for got, exact in ((z, want), (fine.grad, grad)):
        e = helpers.rel_err(got.double().cpu().numpy(), exact.cpu().numpy())
        assert e <= tol, e


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-6), ("tf32x3", helpers.FP32_TOL)])
def test_rows_without_a_rule(precision, tol, cuda):
    """A rulebook built for a coarse grid that does not cover the fine one, found again by a call that names one that does
    (rulebooks are found by fine size, filter and stride): the rows left out get the bias, and no gradient."""
    import ctypes as C

    import sparseconvnet_b200 as scn
    from sparseconvnet_b200 import SCN
    from sparseconvnet_b200._lib import check, lib, sizes
    torch.manual_seed(5)
    x = scn.InputLayer(3, 48, mode=1)([torch.from_numpy(_points(4000, 3, 48, False)), torch.zeros(4000, 1, device=cuda)])
    md, n, two = x.metadata._h, x.features.size(0), sizes([2] * 3)
    cin, cout = 64, 48
    w, bias = torch.randn(8, 1, cin, cout, device=cuda), torch.randn(cout, device=cuda)
    f = torch.randn(n, cout, device=cuda)
    y = f.new_empty(0)
    SCN.Convolution_updateOutput(x.spatial_size, torch.LongTensor([20] * 3), torch.LongTensor([2] * 3), torch.LongTensor([2] * 3),
                                 x.metadata, f, y, torch.randn(8, 1, cout, cin, device=cuda), f.new_empty(0))
    g = torch.randn(y.size(0), cin, device=cuda)
    out, d_in = (torch.full((n, cout), float("nan"), device=cuda) for _ in range(2))
    dw = torch.empty(8, 1, cout, cin, device=cuda)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def ptr(t):
        return C.c_void_p(t.data_ptr())
    wide = sizes([24] * 3), sizes([48] * 3)
    w_back = w.transpose(2, 3).contiguous()
    try:
        scn.set_backward_precision(precision)
        check(lib.scn_deconvolution_forward(md, wide[0], wide[1], two, two, ptr(g), ptr(out), ptr(w), ptr(bias), cin, cout, 1,
                                            {"fp32": 0, "tf32x3": 3}[precision], stream, None))
        check(lib.scn_convolution_backward(md, wide[1], wide[0], two, two, ptr(f), ptr(d_in), ptr(g), ptr(w_back), ptr(dw), None,
                                           cout, cin, 1, stream))
        x.metadata.poll_errors()
    finally:
        scn.set_backward_precision("fp32")
    want, grad = bias.double().expand(n, cout).clone(), torch.zeros(n, cout, dtype=torch.float64, device=cuda)
    seen = torch.zeros(n, dtype=torch.long, device=cuda)
    for r, m in zip(x.metadata.rulebook(1, x.spatial_size, [2] * 3, [2] * 3), w.double()[:, 0]):
        r = r.long()
        seen[r[:, 0]] += 1
        want.index_add_(0, r[:, 0], g.double()[r[:, 1]] @ m)
        grad.index_add_(0, r[:, 0], g.double()[r[:, 1]] @ m)
    assert 0 < int((seen == 0).sum()) < n and int(seen.max()) == 1
    for got, exact in ((out, want), (d_in, grad)):
        e = helpers.rel_err(got.double().cpu().numpy(), exact.cpu().numpy())
        assert e <= tol, e


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-6), ("tf32x3", helpers.FP32_TOL)])
@pytest.mark.parametrize("n", [1, 5000])
def test_windows_of_one_site(n, precision, tol, cuda):
    """Filter and stride 1: the coarse grid has the fine one's size and takes its place while it is read.  Sums of cin products."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(n)
    x = scn.InputLayer(3, 48, mode=1)([torch.from_numpy(_points(n, 3, 48, False)), torch.randn(n, 64, device=cuda)])
    where = x.get_spatial_locations()
    a, b = scn.Convolution(3, 64, 96, 1, 1, False), scn.Deconvolution(3, 96, 32, 1, 1, False)
    try:
        scn.set_precision(precision)
        with torch.no_grad():
            y = a.to(cuda)(x)
            z = b.to(cuda)(y)
        y.metadata.poll_errors()
    finally:
        scn.set_precision("fp32")
    assert torch.equal(y.get_spatial_locations(), where) and torch.equal(z.get_spatial_locations(), where)
    want = x.features.double() @ a.weight.detach().double()[0, 0]
    for got, exact in ((y.features, want), (z.features, y.features.double() @ b.weight.detach().double()[0, 0])):
        e = helpers.rel_err(got.double().cpu().numpy(), exact.cpu().numpy())
        assert e <= tol, e
