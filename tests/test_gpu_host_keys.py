"""Coordinates on the host are checked and packed there: the same sites, rows and errors as for coordinates on the GPU."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _locations(scn, dim, coords, size, mode):
    feats = torch.arange(coords.size(0), dtype=torch.float32, device="cuda")[:, None].contiguous()
    out = scn.InputLayer(dim, torch.LongTensor([size] * dim), mode=mode)([coords, feats])
    return out.get_spatial_locations().cpu(), out.features.cpu()


# pieces of 16384 points are shared out to helper threads
@pytest.mark.parametrize("n", [1, 16383, 16384, 16385, 100003])
@pytest.mark.parametrize("dim,mode", [(2, 0), (3, 3), (4, 4), (1, 2)])
def test_host_and_device_coordinates(n, dim, mode):
    import sparseconvnet_b200 as scn
    g = torch.Generator().manual_seed(n + dim)
    coords = torch.randint(0, 40, (n, dim + 1), generator=g)
    for a, b in zip(_locations(scn, dim, coords, 40, mode), _locations(scn, dim, coords.cuda(), 40, mode)):
        assert torch.equal(a, b)  # whole numbers, and sums of whole numbers below 2^24 or means of the same rows


@pytest.mark.parametrize("row", [0, 16384, 40000])
@pytest.mark.parametrize("value", [-1, 40, 1 << 40])
def test_host_coordinate_out_of_range(row, value):
    import sparseconvnet_b200 as scn
    coords = torch.zeros(40001, 4, dtype=torch.int64)
    coords[row, 1] = value
    with pytest.raises(RuntimeError, match="outside the spatial size"):
        _locations(scn, 3, coords, 40, 3)


# keys of 30 to 33 bits, 36 to 39, 42 to 45, and more than 48 by the coordinates alone, which travel whole; one piece and more
@pytest.mark.parametrize("size", [1000, 4096, 16000, 65000])
@pytest.mark.parametrize("n,batch", [(1, 1), (1025, 8), (16383, 2), (33793, 5)])
@pytest.mark.parametrize("mode", [0, 3])
def test_keys_by_their_bytes(n, batch, size, mode):
    import sparseconvnet_b200 as scn
    g = torch.Generator().manual_seed(n)
    coords = torch.randint(0, size, (n, 4), generator=g)
    coords[:, 3] = torch.randint(0, batch, (n,), generator=g)
    coords[n // 2:] = coords[:n - n // 2].clone()  # every site twice
    for a, b in zip(_locations(scn, 3, coords, size, mode), _locations(scn, 3, coords.cuda(), size, mode)):
        assert torch.equal(a, b)


# One point alone has bits of its key from 48 on, or 47 as the last one without: coordinates of 42 bits, the batch above them.  The
# last point is one that is looked at before the keys are packed, the one before it is not.
@pytest.mark.parametrize("batch", [63, 64, 1 << 14, (1 << 21) - 1])
@pytest.mark.parametrize("row", [19998, 19999])
@pytest.mark.parametrize("mode", [0, 3])
def test_keys_wide_by_their_batch(row, batch, mode):
    import sparseconvnet_b200 as scn
    coords = torch.randint(0, 16000, (20000, 4), generator=torch.Generator().manual_seed(batch))
    coords[:, 3] = torch.arange(20000) // 10000
    coords[9000:10000] = coords[:1000].clone()
    coords[row, 3] = batch
    for a, b in zip(_locations(scn, 3, coords, 16000, mode), _locations(scn, 3, coords.cuda(), 16000, mode)):
        assert torch.equal(a, b)
