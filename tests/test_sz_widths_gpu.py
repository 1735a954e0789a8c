"""Packed bytes of the error-bounded codec where its packer and unpacker branch: planes with rows
of at most 8, at most 16 and more bits side by side in a tile, values off the nearest grid point,
raw tiles between packed ones."""
import numpy as np
import pytest
import torch

from ccbench_b200.ops import sz

pytestmark = pytest.mark.gpu


def _field(kind, shape):
    g = torch.Generator().manual_seed(11)
    f = torch.randn(shape, generator=g)
    if kind == "mixed":      # the scale changes from plane to plane: 3 to 22 bits
        f *= (4.0 ** (torch.arange(shape[0]) % 8)).view(-1, 1, 1)
    elif kind == "rows":     # and inside a plane from one element of eight to the next
        f *= 8.0 ** (torch.arange(shape[2]) % 8 // 2).view(1, 1, -1)
    elif kind == "far":      # large multiples of the step: fp32 rounding picks the farther grid point now and then
        f = f * 0.5 + 8000.0
    elif kind == "raw":      # infinities, NaN and values beyond the integer range, each in a tile of its own
        f[0, 0, 0] = float("inf")
        f[-1, 3, 40] = float("nan")
        f[1, -1, -1] = -3e38
    elif kind == "flat":
        f = torch.zeros(shape)
        f[2] = 1.0
    return f


@pytest.mark.parametrize("kind", ["mixed", "rows", "far", "raw", "flat"])
@pytest.mark.parametrize("shape", [(16, 16, 64), (19, 21, 99), (9, 40, 132), (41, 9, 160)])
def test_bytes_and_values_are_those_of_the_host_codec(kind, shape):
    f = _field(kind, shape)
    eb = 1e-2 if kind != "far" else 1e-3
    buf, used = sz.compress(f.cuda(), eb)
    blob = sz.to_container(buf, shape, eb).cpu().numpy()
    want = sz.encode_cpu(f.numpy(), eb)
    assert np.array_equal(blob, want)
    back = sz.decompress(buf, shape, eb).cpu().numpy()
    assert np.array_equal(back, sz.decode_cpu(want), equal_nan=True)


@pytest.mark.parametrize("shape", [(41, 9, 160), (64, 64, 64)])
@pytest.mark.parametrize("tiles", [[0], [7], list(range(8))])
def test_a_group_given_up_makes_no_container_and_harms_no_other(shape, tiles):
    f = _field("mixed", shape).cuda()
    buf, used = sz.compress(f, 1e-2)
    assert 0 < int(used) < buf.numel()
    back = sz.decompress(buf, shape, 1e-2)
    for t in tiles:
        word = sz.GROUP_STRIDE + 4 * t
        buf[word:word + 4].view(torch.int32).fill_(1 << 24)
    got = sz.decompress(buf, shape, 1e-2)
    tx, ty = -(-shape[2] // sz.TX), -(-shape[1] // sz.TY)
    for t in range(8, 16):   # the tiles of that group may be anything
        z, y, x = t // (tx * ty) * sz.TZ, t // tx % ty * sz.TY, t % tx * sz.TX
        for v in (got, back):
            v[z:z + sz.TZ, y:y + sz.TY, x:x + sz.TX] = 0
    assert torch.equal(got, back)
    for where in (buf, buf.cpu()):
        with pytest.raises(ValueError):
            sz.to_container(where, shape, 1e-2)


@pytest.mark.parametrize("shape", [(192, 192, 256), (190, 191, 255)])
def test_raw_tiles_between_packed_ones_over_several_turns(shape):
    """4608 tiles, 576 groups: more than three a cluster. Runs of raw tiles of every length from none
    to a few groups lie between packed ones, so both scratch buffers of the unpacker and both
    parities of the packer's size exchange are used again around them."""
    g = torch.Generator().manual_seed(3)
    f = torch.randn(shape, generator=g)
    tiles = [-(-shape[0] // 8), -(-shape[1] // 8), -(-shape[2] // 32)]
    hit = (torch.rand(tiles, generator=g) < torch.rand(tiles[0], 1, 1, generator=g)).repeat_interleave(8, 0).repeat_interleave(8, 1).repeat_interleave(32, 2)
    f[hit[:shape[0], :shape[1], :shape[2]]] *= 1e9
    eb = 1e-2
    buf, _ = sz.compress(f.cuda(), eb)
    want = sz.encode_cpu(f.numpy(), eb)
    assert np.array_equal(sz.to_container(buf, shape, eb).cpu().numpy(), want)
    again, s2, e2 = sz.from_container(torch.from_numpy(want).cuda())
    for b in (buf, again):
        back = sz.decompress(b, shape, eb).cpu()
        assert (back - f).abs().max().item() <= eb32(eb)
        assert torch.equal(back, torch.from_numpy(sz.decode_cpu(want)))


def eb32(eb):
    return float(np.float32(eb))
