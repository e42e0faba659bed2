"""k_conv_six: the fp32 mode on tensor cores, operands as three bf16 parts, six products.

Per step of 32 planes the tensor core truncates two sums of 16 products each (2^-23 of them at most), everything else is
rounded to nearest in fp32: the 2-norm of the error stays below 2^-22 of the result's, 2.4e-7, and below that of a chain of
fp32 multiply-adds of a few hundred terms."""
import pytest
import torch

from tests.test_gpu_tile import _points

pytestmark = pytest.mark.gpu
FMA, SIX = 7, 8  # scn_last_conv_kernel


def _exact(x, layer, kind, filt, stride, f, shape):
    want = torch.zeros(shape, dtype=torch.float64, device=f.device)
    if hasattr(layer, "bias"):
        want += layer.bias.double()
    up = type(layer).__name__ == "Deconvolution"
    for r, w in zip(x.metadata.rulebook(kind, x.spatial_size, filt, stride), layer.weight.double()[:, 0]):
        r = r.long().flip(1) if up else r.long()
        want.index_add_(0, r[:, 1], f.double()[r[:, 0]] @ w)
    return want


def _on_six(offsets, cin, cout, rows, side=None):
    """Which layers run on k_conv_six; side: of windows side by side, "fine" rows or "coarse" ones."""
    weights = offsets * cin * cout
    if rows < 512 or (cin <= 16 and rows < 16384) or (cout <= 16 and rows > 131072) or weights < (9000 if offsets < 27 else 6900):
        return False
    if weights * rows < (80e6 if rows >= 2048 else 220e6 if side else 160e6):
        return False
    if side == "coarse":
        return cout > 64 or rows <= 90000
    return side is None or cin * cout >= 20000 or (cin >= 96 and cin * cout >= 8000 and rows >= 40000)


@pytest.mark.parametrize("sign", ["mixed", "one"])
@pytest.mark.parametrize("cin,cout", [(8, 32), (8, 64), (12, 48), (16, 32), (32, 32), (36, 64), (64, 80), (64, 84), (96, 96), (32, 128),
                                      (100, 132), (160, 128), (64, 256)])
@pytest.mark.parametrize("n,split", [(700, None), (1700, None), (8191, None), (20001, None), (8200, "3"), (150000, None)])
def test_as_accurate_as_multiply_adds(n, split, cin, cout, sign, cuda, monkeypatch):
    """Every plane tile and both column layouts, packed and unpacked rows, divided offsets, long and short sums, sums that
    cancel and sums of one sign, where the tensor core's truncation is a bias: against float64 and against the error of
    k_conv_fma (of sums of at most 27 x 160 fp32 products: 1e-5, as in its own test)."""
    import sparseconvnet_b200 as scn
    lib = scn.SCN.lib
    if split:
        monkeypatch.setenv("SCN_SIX_SPLIT", split)
    coords = _points(n, 3, 160 if n < 100000 else 512, n)
    x = scn.InputLayer(3, 512, mode=0)([torch.from_numpy(coords), torch.zeros(len(coords), 1, device=cuda)])
    torch.manual_seed(cin)
    ran = 0
    with torch.no_grad():
        for layer, kind, filt, stride, side in [(scn.SubmanifoldConvolution(3, cin, cout, 3, True), 0, 3, None, None),
                                                (scn.Convolution(3, cin, cout, 2, 2, False), 1, 2, 2, "coarse"),
                                                (scn.Deconvolution(3, cin, cout, 2, 2, False), 1, 2, 2, "fine")]:
            layer.to(cuda)
            layer.weight.normal_()
            if hasattr(layer, "bias"):
                layer.bias.normal_()
            spatial = x.spatial_size // 2 if side == "fine" else x.spatial_size
            f = torch.randn(x.metadata.getNActive(spatial), cin, device=cuda)
            if sign == "one":
                for t in (f, layer.weight) + ((layer.bias,) if hasattr(layer, "bias") else ()):
                    t.abs_()
            errors = []
            for six in ("1", "0"):
                monkeypatch.setenv("SCN_CONV_SIX", six)
                y = layer(scn.SparseConvNetTensor(f, x.metadata, spatial)).features
                if six == "1":
                    expected = _on_six(filt ** 3, cin, cout, len(y), side)
                    assert lib.scn_last_conv_kernel() == (SIX if expected else FMA), (layer, len(y))
                    if not expected:
                        break
                    want = _exact(x, layer, kind, [filt] * 3, stride and [stride] * 3, f, y.shape)
                errors.append(float((y.double() - want).norm() / want.norm()))
            x.metadata.poll_errors()
            if errors:
                ran += 1
                assert errors[0] <= 2.0 ** -22 and errors[1] <= 1e-5 and errors[0] <= 1.05 * errors[1], (layer, errors)
    assert ran or n < 10000


@pytest.mark.parametrize("planes", [32, 96, 160])
def test_largest_part_of_a_product_left_out(planes, cuda, monkeypatch):
    """1.0038986 = h + m + l with m = 2^-8 and l = -2^-17: the terms m l' and l m' that are left out are 2^-24 of every product of
    it with itself, the most there can be, all of one sign.  Beside them an fp32 rounding at the end of each step."""
    import sparseconvnet_b200 as scn
    coords = _points(20001, 3, 160, 1)
    x = scn.InputLayer(3, 160, mode=0)([torch.from_numpy(coords), torch.zeros(len(coords), 1, device=cuda)])
    layer = scn.SubmanifoldConvolution(3, planes, planes, 3, False).to(cuda).requires_grad_(False)
    layer.weight.fill_(1.0038986)
    f = torch.full((len(coords), planes), 1.0038986, device=cuda)
    y = layer(scn.SparseConvNetTensor(f, x.metadata, x.spatial_size)).features
    assert scn.SCN.lib.scn_last_conv_kernel() == SIX
    want = _exact(x, layer, 0, [3, 3, 3], None, f, y.shape)
    assert float((y.double() - want).norm() / want.norm()) <= 2.0 ** -22
    assert float(((y.double() - want) / want).abs().max()) <= 2.0 ** -21


@pytest.mark.parametrize("case", ["inf", "nan", "huge", "tiny", "tiny weights", "inf weight", "zeros"])
@pytest.mark.parametrize("cin,cout,n", [(32, 32, 5000), (40, 136, 5000)])
def test_values_the_parts_cannot_hold(case, cin, cout, n, cuda, monkeypatch):
    """Infinities, NaN and the ends of the range: as fp32 multiply-adds in the order of k_conv_fma give them."""
    import sparseconvnet_b200 as scn
    coords = _points(n, 3, 60, 3)
    x = scn.InputLayer(3, 60, mode=0)([torch.from_numpy(coords), torch.zeros(len(coords), 1, device=cuda)])
    torch.manual_seed(1)
    layer = scn.SubmanifoldConvolution(3, cin, cout, 3, True).to(cuda).requires_grad_(False)
    f = torch.randn(len(coords), cin, device=cuda)
    if case in ("inf", "nan"):
        f[17, 3] = float(case)
    elif case == "huge":
        f[5] = 2.9e38
    elif case == "tiny":
        f *= 1e-38
    elif case == "tiny weights":
        f *= 1e-14
        layer.weight *= 1e-14
    elif case == "inf weight":
        layer.weight[13, 0, 2, 1] = float("inf")
    else:
        f.zero_()
    outs = []
    for six, knob in (("1", "SCN_SIX_SPLIT"), ("0", "SCN_FMA_SPLIT")):
        monkeypatch.setenv("SCN_CONV_SIX", six)
        monkeypatch.setenv(knob, "1")
        with torch.no_grad():
            outs.append(layer(scn.SparseConvNetTensor(f, x.metadata, x.spatial_size)).features)
        assert scn.SCN.lib.scn_last_conv_kernel() == (SIX if six == "1" else FMA)
    x.metadata.poll_errors()
    got, want = outs
    if case == "inf weight":  # k_conv_fma multiplies the rows without a rule by it as well
        finite = torch.isfinite(want)
        assert torch.equal(got[finite], want[finite]) and not torch.isfinite(got[:, 1]).all()
    else:
        assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))


@pytest.mark.parametrize("cin,cout,n,split", [(32, 32, 9000, "1"), (40, 48, 3000, "3"), (100, 136, 700, None), (64, 128, 9000, None)])
def test_an_infinity_spoils_its_own_rows_only(cin, cout, n, split, cuda, monkeypatch):
    """One infinite weight of an offset that some rows have: the others, and the planes beside it, as float64 gives them, with
    the offsets whole and divided (sums of 27 x 100 fp32 products: 1e-5 as in the multiply-adds' own test)."""
    import sparseconvnet_b200 as scn
    if split:
        monkeypatch.setenv("SCN_SIX_SPLIT", split)
    coords = _points(n, 3, 160, n)
    x = scn.InputLayer(3, 160, mode=0)([torch.from_numpy(coords), torch.zeros(len(coords), 1, device=cuda)])
    torch.manual_seed(n)
    layer = scn.SubmanifoldConvolution(3, cin, cout, 3, True).to(cuda).requires_grad_(False)
    layer.bias.normal_()
    f = torch.randn(len(coords), cin, device=cuda)
    monkeypatch.setenv("SCN_CONV_SIX", "1")
    layer(scn.SparseConvNetTensor(f, x.metadata, x.spatial_size))
    want = _exact(x, layer, 0, [3, 3, 3], None, f, (len(coords), cout))
    book = x.metadata.rulebook(0, x.spatial_size, [3, 3, 3], None)
    k = max((k for k in range(27) if k != 13), key=lambda k: len(book[k]))
    layer.weight[k, 0, 2, 1] = float("inf")
    y = layer(scn.SparseConvNetTensor(f, x.metadata, x.spatial_size)).features
    assert scn.SCN.lib.scn_last_conv_kernel() == SIX
    x.metadata.poll_errors()
    hit = torch.zeros(len(coords), cout, dtype=torch.bool, device=cuda)
    hit[book[k].long()[:, 1], 1] = True
    assert 0 < int(hit.sum()) < len(coords) and torch.equal(hit, ~torch.isfinite(y))
    assert float((y.double() - want)[~hit].abs().max() / want.abs().max()) <= 1e-5


@pytest.mark.parametrize("case", ["4-D", "down", "up"])
def test_an_infinity_on_other_tables(case, cuda, monkeypatch):
    """81 offsets in four mask words, coarse rows, tiles of one offset with rows left over: the bits of k_conv_fma."""
    import sparseconvnet_b200 as scn
    dim, cin, cout = (4, 32, 48) if case == "4-D" else (3, 160, 132)
    coords = _points(20000, dim, 24 if dim == 4 else 90, 2)
    x = scn.InputLayer(dim, 24 if dim == 4 else 90, mode=0)([torch.from_numpy(coords), torch.zeros(len(coords), 4, device=cuda)])
    torch.manual_seed(dim)
    layer = {"4-D": lambda: scn.SubmanifoldConvolution(4, cin, cout, 3, True), "down": lambda: scn.Convolution(3, cin, cout, 2, 2, True),
             "up": lambda: scn.Deconvolution(3, cin, cout, 2, 2, True)}[case]().to(cuda).requires_grad_(False)
    if case == "up":
        x = scn.Convolution(3, 4, 4, 2, 2, False).to(cuda).requires_grad_(False)(x)
    f = torch.randn(x.features.size(0), cin, device=cuda)
    f[5, 3] = float("inf")
    outs = []
    for six, knob in (("1", "SCN_SIX_SPLIT"), ("0", "SCN_FMA_SPLIT")):
        monkeypatch.setenv("SCN_CONV_SIX", six)
        monkeypatch.setenv(knob, "1")
        outs.append(layer(scn.SparseConvNetTensor(f, x.metadata, x.spatial_size)).features)
        assert scn.SCN.lib.scn_last_conv_kernel() == (SIX if six == "1" else FMA)
    x.metadata.poll_errors()
    assert 0 < int((~torch.isfinite(outs[1])).sum()) < outs[1].numel() // 2
    assert torch.equal(*(torch.nan_to_num(y, nan=7.0) for y in outs))


@pytest.mark.parametrize("small", [1e-30, 1e-35, 1e-37])
@pytest.mark.parametrize("cin,cout", [(24, 32), (32, 32), (40, 136)])
def test_small_values_beside_ordinary_ones(small, cin, cout, cuda):
    """A sample of small values beside an ordinary one, output planes of small weights beside ordinary ones: each as accurate by
    itself (results of 1e-36 and above, where fp32's own rounding of subnormal numbers is below 2^-22 of them)."""
    import sparseconvnet_b200 as scn
    coords = _points(20001, 3, 80, 9)
    coords[:, 3] = coords[:, 0] >= 40  # (samples share no rule)
    x = scn.InputLayer(3, 80, mode=0)([torch.from_numpy(coords), torch.zeros(len(coords), 1, device=cuda)])
    torch.manual_seed(cin)
    layer = scn.SubmanifoldConvolution(3, cin, cout, 3, False).to(cuda).requires_grad_(False)
    layer.weight.normal_()
    layer.weight[..., 8:12] *= small
    f = torch.randn(len(coords), cin, device=cuda)
    tiny = torch.from_numpy(coords[:, 3] == 1).to(cuda)
    f[tiny] *= small
    y = layer(scn.SparseConvNetTensor(f, x.metadata, x.spatial_size)).features
    assert scn.SCN.lib.scn_last_conv_kernel() == SIX
    x.metadata.poll_errors()
    want = _exact(x, layer, 0, [3, 3, 3], None, f, y.shape)
    plane = torch.zeros(cout, dtype=torch.bool, device=cuda)
    plane[8:12] = True
    for rows, planes in ((~tiny, ~plane), (tiny, ~plane), (~tiny, plane)):
        got, exact = y.double()[rows][:, planes], want[rows][:, planes]
        assert float(exact.norm()) > 0
        e = (got - exact).norm(dim=1) / exact.norm(dim=1).clamp(min=1e-37)
        assert float(e.max()) <= 2.0 ** -20 and float((got - exact).norm() / exact.norm()) <= 2.0 ** -22


@pytest.mark.parametrize("cin,cout", [(32, 48), (24, 160)])
def test_weights_of_this_call(cin, cout, cuda):
    """A weight written through .data, which leaves its version as it is, counts from the next call on."""
    import sparseconvnet_b200 as scn
    coords = _points(6000, 3, 60, 4)
    x = scn.InputLayer(3, 60, mode=0)([torch.from_numpy(coords), torch.randn(len(coords), cin, device=cuda)])
    layer = scn.SubmanifoldConvolution(3, cin, cout, 3, False).to(cuda)
    with torch.no_grad():
        one = layer(x).features
        assert scn.SCN.lib.scn_last_conv_kernel() == SIX
        layer.weight.data.mul_(2)
        assert torch.equal(layer(x).features, 2 * one)


@pytest.mark.parametrize("n,inf", [(700, False), (20000, False), (20000, True)])
def test_batchnorm_and_join_in_front(n, inf, cuda):
    """In the pass that splits the rows, and where they are multiplied unsplit: the same bits as the layers one by one."""
    import sparseconvnet_b200 as scn
    torch.manual_seed(n)

    def block(planes):
        return scn.Sequential().add(scn.BatchNormLeakyReLU(planes, leakiness=0.2)).add(scn.SubmanifoldConvolution(3, planes, 32, 3, True))
    net = scn.Sequential().add(scn.ConcatTable().add(scn.Identity()).add(block(32))).add(scn.JoinTable()).add(block(64)).to(cuda).eval()
    for m in net.modules():
        if isinstance(m, scn.BatchNormalization):
            for t in (m.running_mean, m.running_var, m.weight, m.bias):
                torch.nn.init.uniform_(t, 0.3, 1.0)
    coords = _points(n, 3, 120, n)
    feats = torch.randn(len(coords), 32, device=cuda)
    if inf:
        feats[7, 3] = float("inf")
    outs = []
    try:
        for fuse in (False, True):
            scn.Sequential.fuse = fuse
            with torch.no_grad():
                outs.append(net(scn.InputLayer(3, 120, mode=0)([torch.from_numpy(coords), feats])).features)
    finally:
        scn.Sequential.fuse = True
    assert not inf or 0 < int((~torch.isfinite(outs[0])).sum()) < outs[0].numel() // 2
    assert torch.equal(*(torch.nan_to_num(y, nan=7.0) for y in outs))


def test_bounded_wait_runs_out(cuda):
    """One barrier arrival left out: the kernel returns by itself, the host learns of it, the next call is right."""
    import sparseconvnet_b200 as scn
    from sparseconvnet_b200._lib import ScnError, lib
    coords = _points(20000, 3, 96, 5)
    layer = scn.SubmanifoldConvolution(3, 96, 96, 3, False).to(cuda)
    with torch.no_grad():
        x = scn.InputLayer(3, 96, mode=0)([torch.from_numpy(coords), torch.randn(len(coords), 96, device=cuda)])
        good = layer(x).features.clone()
        assert lib.scn_last_conv_kernel() == SIX
        x.metadata.poll_errors()
        assert lib.scn_test_drop_barrier_arrival() == 0
        layer(x)
        torch.cuda.synchronize()
        with pytest.raises(ScnError, match="bounded wait"):
            x.metadata.poll_errors()
        assert torch.equal(layer(x).features, good)
        x.metadata.poll_errors()


@pytest.mark.parametrize("kind,cin,cout,n", [("submanifold", 64, 96, 9000), ("submanifold", 64, 96, 1600), ("submanifold", 64, 64, 3000),
                                             ("down", 96, 160, 9000), ("up", 160, 160, 30000)])
def test_without_memory_for_the_parts(kind, cin, cout, n, cuda, monkeypatch):
    """Every allocation of a layer whose rulebook is there fails in turn: where the operands' parts do not fit, or the row order of
    a level that k_conv_fma takes as it is, that kernel's result; an error only for what it needs as well."""
    import sparseconvnet_b200 as scn
    from sparseconvnet_b200._lib import ScnError, lib
    torch.manual_seed(n)
    coords = torch.from_numpy(_points(n, 3, 160, n)).to(cuda)
    make, small = ((lambda a, b: scn.SubmanifoldConvolution(3, a, b, 3, True),) * 2 if kind == "submanifold" else
                   (lambda a, b: scn.Convolution(3, a, b, 2, 2, True),) * 2 if kind == "down" else
                   (lambda a, b: scn.Deconvolution(3, a, b, 2, 2, True), lambda a, b: scn.Convolution(3, a, b, 2, 2, True)))
    layer, first = make(cin, cout).to(cuda).requires_grad_(False), small(4, 4).to(cuda).requires_grad_(False)
    feats = torch.randn(len(coords), cin, device=cuda)

    def run(which, six):
        monkeypatch.setenv("SCN_CONV_SIX", six)
        x = scn.InputLayer(3, 160, mode=1)([coords, feats[:, :4].contiguous()])
        y = first(x)  # the rulebook, on a kernel without tiles
        rows = y.features.size(0) if kind == "up" else x.features.size(0)
        z = scn.SparseConvNetTensor(feats[:rows], x.metadata, y.spatial_size if kind == "up" else x.spatial_size)
        lib.scn_test_fail_allocation(which)
        try:
            out = layer(z).features
        finally:
            left = lib.scn_test_fail_allocation(0)
        x.metadata.poll_errors()
        return out, lib.scn_last_conv_kernel() == SIX, left
    want, on_six, _ = run(0, "1")
    plain, on_fma, _ = run(0, "0")
    assert on_six and not on_fma
    recovered, failed = 0, 0
    for which in range(1, 40):
        try:
            out, six, left = run(which, "1")
        except ScnError as e:
            assert "out of memory" in str(e)
            failed += 1
            continue
        assert torch.equal(out, want if six else plain), which
        if left:
            break
        assert not six
        recovered += 1
    assert left and recovered >= 2 and (failed == 0) == (len(want) < 2048)
