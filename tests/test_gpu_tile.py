"""k_conv_tile and the row order it packs its tiles by, against the fp32 kernels (themselves checked against the
reference's results in test_gpu_parity.py).

Tolerances relative to the largest output: the three-term form drops m m' and what h + m leaves of x, 2^-17 of a product
each, so 2^-16 of the largest sum of |products|, which stays below 4 of the largest output for these random sums: 1e-4
(the fp32 bar).  One bf16 product: 2^-8 per product, averaging to 1e-2."""
import numpy as np
import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu

TOL = {"tf32x3": helpers.FP32_TOL, "tf32": helpers.FP32_TOL, "bf16": helpers.TC_TOL}


def _points(n, dim, size, seed):
    rng = np.random.default_rng(seed)
    pts = rng.integers(0, size, (n, dim))
    if n > 200:  # a wavy surface: masks repeat as they do on scans
        pts[:, dim - 1] = size // 2 + size // 5 * np.sin(pts[:, 0] / 6.0) + rng.integers(0, 2, n)
    pts = np.unique(pts, axis=0)[rng.permutation(len(np.unique(pts, axis=0)))]
    return np.concatenate([pts, rng.integers(0, 2, (len(pts), 1))], axis=1)


def _compare(layers, coords, dim, size, cin, precision, cuda, mode=3):
    import sparseconvnet_b200 as scn
    rng = np.random.default_rng(cin)
    feats = torch.from_numpy(rng.standard_normal((coords.shape[0], cin)).astype(np.float32)).to(cuda)
    try:
        with torch.no_grad():
            x = scn.InputLayer(dim, size, mode=mode)([torch.from_numpy(coords), feats])
            for layer in layers:
                scn.set_precision("fp32")
                want = layer.to(cuda)(x)
                scn.set_precision(precision)
                got = layer(x)
                assert scn.SCN.lib.scn_last_conv_kernel() == 6, "not on k_conv_tile"
                again = layer(x)
                x.metadata.poll_errors()
                assert got.features.shape == want.features.shape
                assert torch.equal(got.features, again.features), "not the same twice"
                e = helpers.rel_err(got.features.cpu().numpy(), want.features.cpu().numpy())
                assert e <= TOL[precision], (layer, precision, coords.shape[0], e)
                x = want
    finally:
        scn.set_precision("fp32")


@pytest.mark.parametrize("precision", ["tf32x3", "bf16", "tf32"])
@pytest.mark.parametrize("cin,cout", [(32, 32), (16, 16), (8, 24), (24, 40), (48, 64), (64, 72), (96, 96), (80, 160),
                                      (128, 256), (320, 8)])
def test_plane_counts(cin, cout, precision, cuda):
    import sparseconvnet_b200 as scn
    torch.manual_seed(cin + cout)
    sc = scn.SubmanifoldConvolution(3, cin, cout, 3, True)
    sc.bias.data.normal_()
    _compare([sc], _points(9001, 3, 72, 1), 3, 72, cin, precision, cuda)


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 257, 4095, 4097, 60001])
@pytest.mark.parametrize("cin,cout", [(32, 32), (64, 96)])
def test_row_counts(n, cin, cout, cuda):
    import sparseconvnet_b200 as scn
    torch.manual_seed(n)
    layers = [scn.SubmanifoldConvolution(3, cin, cout, 3, False), scn.Convolution(3, cout, 64, 2, 2, True),
              scn.SubmanifoldConvolution(3, 64, 64, 3, False), scn.Deconvolution(3, 64, 32, 2, 2, False)]
    _compare(layers, _points(n, 3, 160, n), 3, 160, cin, "tf32x3", cuda, mode=0 if n < 300 else 3)


@pytest.mark.parametrize("dim,filter_size,stride", [(1, 3, 2), (2, 3, 2), (2, 5, 3), (3, 1, 1), (4, 3, 2), (3, 5, 2)])
def test_filters(dim, filter_size, stride, cuda):
    """1 to 125 filter offsets: one to five sort digits, one and four mask words, keys that join offsets."""
    import sparseconvnet_b200 as scn
    size = {1: 4001, 2: 182, 3: 63, 4: 23}[dim]
    size = (size - filter_size) // stride * stride + filter_size
    torch.manual_seed(dim)
    layers = [scn.SubmanifoldConvolution(dim, 32, 48, filter_size, False)]
    if filter_size > 1:
        layers += [scn.Convolution(dim, 48, 32, filter_size, stride, False), scn.Deconvolution(dim, 32, 16, filter_size, stride, False)]
    pts = _points(14000, dim, size, dim)
    pts[:, :dim] = np.clip(pts[:, :dim], 0, size - 1)
    _compare(layers, pts, dim, size, 32, "tf32x3", cuda)


@pytest.mark.parametrize("split", ["1", "2", "5", "16"])
@pytest.mark.parametrize("precision", ["tf32x3", "bf16"])
@pytest.mark.parametrize("n", [700, 30000])
def test_splits(split, precision, n, cuda, monkeypatch):
    import sparseconvnet_b200 as scn
    monkeypatch.setenv("SCN_TILE_SPLIT", split)
    torch.manual_seed(n)
    layers = [scn.SubmanifoldConvolution(3, 64, 64, 3, True), scn.SubmanifoldConvolution(3, 64, 128, 3, False),
              scn.Convolution(3, 128, 96, 2, 2, False)]
    _compare(layers, _points(n, 3, 120, 7), 3, 120, 64, precision, cuda)


@pytest.mark.parametrize("cin,cout", [(8, 8), (12, 16), (24, 32), (32, 36), (36, 64), (64, 96), (100, 160), (64, 224)])
@pytest.mark.parametrize("n,split", [(1, None), (31, None), (900, "3"), (8191, None), (8200, "7"), (60001, None)])
def test_fp32_tiles(n, split, cin, cout, cuda, monkeypatch):
    """k_conv_fma (fp32) against a float64 product over the exported rulebook: packed and unpacked rows, both tile heights,
    every plane tile, with and without divided offsets.  Sums of at most 27 x 100 fp32 products: 2700 x 2^-24 of the
    largest sum of magnitudes at the very worst, 2^-24 sqrt(2700) in practice; 1e-5."""
    import sparseconvnet_b200 as scn
    monkeypatch.setenv("SCN_CONV_SIX", "0")
    if split:
        monkeypatch.setenv("SCN_FMA_SPLIT", split)
    coords = _points(n, 3, 160, n)
    x = scn.InputLayer(3, 160, mode=0)([torch.from_numpy(coords), torch.zeros(len(coords), 1, device=cuda)])
    torch.manual_seed(cin)
    layers = [(scn.SubmanifoldConvolution(3, cin, cout, 3, True), 0, [3, 3, 3], None, x.spatial_size),
              (scn.Convolution(3, cin, cout, 2, 2, True), 1, [2, 2, 2], [2, 2, 2], x.spatial_size),
              (scn.Deconvolution(3, cin, cout, 2, 2, False), 1, [2, 2, 2], [2, 2, 2], torch.LongTensor([80, 80, 80]))]
    with torch.no_grad():
        for layer, kind, filt, stride, spatial in layers:
            layer.to(cuda)
            if hasattr(layer, "bias"):
                layer.bias.normal_()
            f = torch.randn(x.metadata.getNActive(spatial), cin, device=cuda)
            y = layer(scn.SparseConvNetTensor(f, x.metadata, spatial)).features
            assert scn.SCN.lib.scn_last_conv_kernel() == 7 or y.size(0) == 0, "not on k_conv_fma"
            want = torch.zeros(y.shape, dtype=torch.float64, device=cuda)
            if hasattr(layer, "bias"):
                want += layer.bias.double()
            for r, w in zip(x.metadata.rulebook(kind, x.spatial_size, filt, stride), layer.weight.double()[:, 0]):
                r = r.long() if not isinstance(layer, scn.Deconvolution) else r.long().flip(1)
                want.index_add_(0, r[:, 1], f.double()[r[:, 0]] @ w)
            e = helpers.rel_err(y.double().cpu().numpy(), want.cpu().numpy())
            assert e <= 1e-5, (layer, e)
            x.metadata.poll_errors()


@pytest.mark.parametrize("precision", ["tf32x3", "bf16"])
@pytest.mark.parametrize("n,planes", [(1, 8), (700, 24), (9000, 32), (9000, 64)])
def test_batchnorm_in_front(n, planes, precision, cuda):
    """A residual block's BatchNorm in front of its convolution rides in the pass that splits the rows: the same bits."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(planes)
    net = scn.Sequential()
    for _ in range(2):
        net.add(scn.ConcatTable().add(scn.Identity()).add(
            scn.Sequential().add(scn.BatchNormLeakyReLU(planes, leakiness=0.2)).add(scn.SubmanifoldConvolution(3, planes, planes, 3, True))
            .add(scn.BatchNormReLU(planes)).add(scn.SubmanifoldConvolution(3, planes, planes, 3, False)))).add(scn.AddTable())
    for m in net.modules():
        if isinstance(m, scn.BatchNormalization):
            for t in (m.running_mean, m.running_var, m.weight, m.bias):
                torch.nn.init.uniform_(t, 0.3, 1.0)
    net.to(cuda).eval()
    coords = _points(n, 3, 120, n)
    feats = torch.randn(len(coords), planes, device=cuda)
    outs = []
    try:
        scn.set_precision(precision)
        for fuse in (False, True):
            scn.Sequential.fuse = fuse
            with torch.no_grad():
                outs.append(net(scn.InputLayer(3, 120, mode=0)([torch.from_numpy(coords), feats])).features)
    finally:
        scn.set_precision("fp32")
        scn.Sequential.fuse = True
    assert torch.equal(*outs)


@pytest.mark.parametrize("precision,planes", [("tf32x3", 16), ("tf32x3", 48), ("tf32x3", 64), ("bf16", 32), ("bf16", 64)])
@pytest.mark.parametrize("n,split", [(1, "1"), (700, "1"), (700, "3"), (20000, None)])
def test_split_rows_left_for_the_next_layer(n, split, planes, precision, cuda, monkeypatch):
    """A convolution's result in split form, from its own store or from the sum of its parts: the next layer gives the same
    bits with it as without, and does not use it once the features have changed."""
    import sparseconvnet_b200 as scn
    if split:
        monkeypatch.setenv("SCN_TILE_SPLIT", split)
    torch.manual_seed(planes)
    a, b = (scn.SubmanifoldConvolution(3, planes, planes, 3, True).to(cuda) for _ in range(2))
    coords = _points(n, 3, 120, n)
    try:
        scn.set_precision(precision)
        with torch.no_grad():
            x = scn.InputLayer(3, 120, mode=0)([torch.from_numpy(coords), torch.randn(len(coords), planes, device=cuda)])
            y, z = a.forward(x, want_split=True), a(x)
            assert y.split is not None and z.split is None
            assert torch.equal(y.features, z.features)
            assert torch.equal(b(y).features, b(z).features)
            y.features.mul_(2)
            z.features.mul_(2)
            assert torch.equal(b(y).features, b(z).features)
            x.metadata.poll_errors()
    finally:
        scn.set_precision("fp32")


@pytest.mark.parametrize("precision", ["tf32x3", "bf16"])
def test_split_rows_and_a_hook_on_the_next_layer(precision, cuda):
    """A forward pre-hook that changes the features through .data, which leaves their version as it is, and an input that
    only looks like a SparseConvNetTensor: the next layer computes with the features as they are."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(0)
    net = scn.Sequential().add(scn.SubmanifoldConvolution(3, 32, 32, 3, True)).add(scn.BatchNormReLU(32)).add(
        scn.SubmanifoldConvolution(3, 32, 48, 3, True)).to(cuda).eval()

    class Looks:
        def __init__(self, x):
            self.features, self.metadata, self.spatial_size = x.features, x.metadata, x.spatial_size
    try:
        scn.set_precision(precision)
        with torch.no_grad():
            coords = _points(5000, 3, 60, 0)
            x = scn.InputLayer(3, 60, mode=0)([torch.from_numpy(coords), torch.randn(len(coords), 32, device=cuda)])
            plain = net(x).features.clone()
            mid = net[1](net[0](x))
            mid.features.mul_(3)
            want = net[2](mid).features
            assert torch.equal(net[2](Looks(mid)).features, want)

            def triple(module, args):
                args[0].features.data.mul_(3)
            handle = net[2].register_forward_pre_hook(triple)
            got = net(x).features
            handle.remove()
            assert torch.equal(got, want) and not torch.equal(got, plain)
            assert torch.equal(net(x).features, plain)
    finally:
        scn.set_precision("fp32")


@pytest.mark.parametrize("precision", ["fp32", "tf32x3", "bf16"])
@pytest.mark.parametrize("n", [300, 30000])
@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 96)])
def test_scale_and_shift_anywhere(n, cin, cout, precision, cuda):
    """Scale and shift of a BatchNorm in front of and behind a convolution as slices that start at any multiple of four
    bytes: the same bits as from arrays of their own."""
    import sparseconvnet_b200 as scn
    from sparseconvnet_b200 import SCN
    torch.manual_seed(n)
    coords = _points(n, 3, 120, n)
    x = scn.InputLayer(3, 120, mode=0)([torch.from_numpy(coords), torch.randn(len(coords), cin, device=cuda)])
    w, three = torch.randn(27, 1, cin, cout, device=cuda), torch.LongTensor([3] * 3)
    post, pre = torch.rand(2, cout, device=cuda) + 0.5, torch.rand(2, cin, device=cuda) + 0.5
    try:
        scn.set_precision(precision)
        results = []
        for offset in (0, 1, 2, 3):
            def place(v):
                return torch.empty(offset + v.numel(), device=cuda)[offset:].copy_(v)
            out, both = (x.features.new_empty(0) for _ in range(2))
            epilogue = (place(post[0]), place(post[1]), 0.25)
            SCN.SubmanifoldConvolution_updateOutput(x.spatial_size, three, x.metadata, x.features, out, w, None, epilogue=epilogue)
            half = cin // 2
            assert SCN.SubmanifoldConvolution_joined(
                x.spatial_size, three, x.metadata, [x.features[:, :half].contiguous(), x.features[:, half:].contiguous()], both, w,
                None, prologue=(place(pre[0]), place(pre[1]), 0.5), epilogue=epilogue) is not None
            results.append((out, both))
        x.metadata.poll_errors()
        for out, both in results[1:]:
            assert torch.equal(out, results[0][0]) and torch.equal(both, results[0][1])
    finally:
        scn.set_precision("fp32")


@pytest.mark.parametrize("n", [1, 127, 128, 129, 3000])
@pytest.mark.parametrize("dim,filter_size", [(1, 1), (3, 3), (1, 31), (2, 5), (1, 33), (2, 7)])
def test_rows_in_their_own_order(n, dim, filter_size, cuda):
    """Tiles of levels too small to sort, up to 32 offsets (one word of a mask) and above: against float64."""
    import sparseconvnet_b200 as scn
    coords = _points(n, dim, 8192 if dim == 1 else 200 if dim == 2 else 40, n)
    torch.manual_seed(n)
    layer = scn.SubmanifoldConvolution(dim, 16, 16, filter_size, True).to(cuda)
    size = torch.LongTensor([8192 if dim == 1 else 200 if dim == 2 else 40] * dim)
    try:
        scn.set_precision("tf32x3")
        with torch.no_grad():
            x = scn.InputLayer(dim, size, mode=0)([torch.from_numpy(coords), torch.randn(len(coords), 16, device=cuda)])
            y = layer(x).features
            x.metadata.poll_errors()
            want = torch.zeros(len(coords), 16, dtype=torch.float64, device=cuda) + layer.bias.double()
            for r, w in zip(x.metadata.rulebook(0, size, [filter_size] * dim, None), layer.weight.double()[:, 0]):
                r = r.long().to(cuda)
                want.index_add_(0, r[:, 1], x.features.double()[r[:, 0]] @ w)
            # (three bf16 terms of a product: 2^-16 of it is left out at most)
            assert float((y.double() - want).norm() / want.norm()) <= 2.0 ** -16
    finally:
        scn.set_precision("fp32")


# one slice and several, one accumulator range and three, one and two CTAs per SM, offsets divided and not, few stages and many
@pytest.mark.parametrize("precision,cin,cout,n", [
    ("tf32x3", 32, 32, 20000), ("tf32x3", 224, 224, 700), ("bf16", 64, 64, 9000), ("fp32", 16, 32, 20000), ("fp32", 64, 64, 9000),
    ("fp32", 160, 160, 3000)])
def test_giving_up_in_every_form(precision, cin, cout, n, cuda):
    """One barrier arrival left out in k_conv_tile's or k_conv_six's first CTA, at a step from which all its roles run dry: the kernel
    ends by itself, the host learns of it, and nothing of it is left for the next call."""
    import sparseconvnet_b200 as scn
    from sparseconvnet_b200._lib import ScnError, lib
    coords = _points(n, 3, 200, n)
    layer = scn.SubmanifoldConvolution(3, cin, cout, 3, True).to(cuda)
    try:
        scn.set_precision(precision)
        with torch.no_grad():
            x = scn.InputLayer(3, 200, mode=3)([torch.from_numpy(coords), torch.randn(len(coords), cin, device=cuda)])
            good = layer(x).features
            assert lib.scn_last_conv_kernel() == (8 if precision == "fp32" else 6)
            x.metadata.poll_errors()
            assert lib.scn_test_drop_barrier_arrival() == 0
            layer(x)
            torch.cuda.synchronize()
            with pytest.raises(ScnError, match="bounded wait"):
                x.metadata.poll_errors()
            for _ in range(3):
                assert torch.equal(layer(x).features, good)
            x.metadata.poll_errors()
    finally:
        scn.set_precision("fp32")
