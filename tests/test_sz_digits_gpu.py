"""Unpacking of fields of many tiles, whose prefix sums run on the tensor cores in digits of seven and eight bits:
residuals on either side of each number of digits, in first planes and in others, and the largest sums."""
import pytest
import torch

from ccbench_b200.ops import sz

pytestmark = pytest.mark.gpu

EB = 2.0 ** -6


def _residuals(first, other, g):
    """One tile [8, 8, 32]: residuals of `other` bits (zig-zag), `first` bits in the corner value."""
    half = 1 << other >> 1
    d = torch.randint(-half, max(half, 1), (8, 8, 32), generator=g) if other else torch.zeros(8, 8, 32, dtype=torch.int64)
    if other:
        d.view(-1)[1 + torch.randperm(2047, generator=g)[:2]] = torch.tensor([-half, half - 1])
    if first:
        d[0, 0, 0] = -(1 << first >> 1)
    return d


@pytest.mark.parametrize("shape", [(160, 168, 256), (161, 163, 260), (200, 201, 257)])   # lines on 32 bytes, on 16, anywhere
def test_every_width_of_residuals_comes_back(shape):
    g = torch.Generator().manual_seed(5)
    kinds = [_residuals(first, other, g) for first in (0, 8, 9, 15, 16, 22) for other in (0, 1, 2, 7, 8, 9, 13, 14, 15, 16)]
    kinds += [torch.full((8, 8, 32), -128), torch.full((8, 8, 32), 127), _residuals(22, 8, g)]   # sums of 2048 residuals
    codes = torch.stack([k.cumsum(0).cumsum(1).cumsum(2) for k in kinds])
    codes = codes[codes.abs().amax((1, 2, 3)) < 1 << 21]
    assert len(codes) > 40
    tz, ty, tx = (-(-n // t) for n, t in zip(shape, (8, 8, 32)))
    pick = torch.randint(0, len(codes), (tz, ty, tx), generator=g)
    q = codes[pick].permute(0, 3, 1, 4, 2, 5).reshape(8 * tz, 8 * ty, 32 * tx)[:shape[0], :shape[1], :shape[2]]
    step = torch.tensor(2 * EB, dtype=torch.float32) * (1 - 2.0 ** -10)   # what the decoder multiplies with, exact here
    field = (q.float() * step).cuda()
    buf, _ = sz.compress(field, EB)
    assert torch.equal(sz.decompress(buf, shape, EB), field)
    tiles = buf.view(-1, sz.GROUP_STRIDE)[:, :sz.GROUP_HEADER].contiguous().view(torch.int32)
    assert int((tiles == sz.TILE_CAP).sum()) == 0 and int(((tiles > 2816) & (tiles <= 4128)).sum()) > 0 and int((tiles[tiles > 0] <= 2816).sum()) > 0


def test_a_buffer_on_four_bytes_is_unpacked_where_it_lies():
    shape = (160, 168, 256)
    f = torch.randn(shape, generator=torch.Generator().manual_seed(1)).cuda().cumsum(2)
    buf, _ = sz.compress(f, 1e-2)
    want = sz.decompress(buf, shape, 1e-2)
    moved = torch.empty(buf.numel() + 16, dtype=torch.uint8, device="cuda")[4:4 + buf.numel()]
    moved.copy_(buf)
    assert torch.equal(sz.decompress(moved, shape, 1e-2), want)


@pytest.mark.parametrize("nx", [0, 4, 5])   # off a whole number of tiles: lines on 32 bytes, on 16, anywhere
def test_tiles_packed_in_halves_end_where_they_should(nx):
    """Codes on either side of where two residuals no longer share a word: far from a tile's first code, first
    codes of more than 8, 16 and 22 bits, in the first plane and in the last."""
    g = torch.Generator().manual_seed(9)
    tiles = []
    for corner in (0, 127, -128, 128, 31999, -32000, 32000, (1 << 21) - 4097, (1 << 21) - 4095, -(1 << 21) - 5, (1 << 22) - 3):
        for spread in (3, 4093, 4094, 4095, 40000):
            t = torch.randint(-1, 2, (8, 8, 32), generator=g) + corner
            t[0, 0, 0] = corner
            t[0 if spread % 2 else 7, 5, 31] = corner + spread if corner < 0 or spread < 5 else corner - spread
            tiles.append(t)
    alternating = torch.where((torch.arange(8)[:, None, None] + torch.arange(8)[:, None] + torch.arange(32)) % 2 == 0, 4094, -4094)
    alternating[0, 0, 0] = 0
    tiles.append(alternating)   # residuals of 8 x 4094
    tiles.append(torch.zeros(8, 8, 32, dtype=torch.int64))
    q = torch.cat(tiles, dim=2)
    step = torch.tensor(2 * EB, dtype=torch.float32) * (1 - 2.0 ** -10)
    f = q.float() * step
    f += (torch.rand(f.shape, generator=g) - 0.5) * step * (q.abs() < 4000)   # off the grid, near ties among them
    f = f[:, :, :f.shape[2] - (32 - nx if nx else 0)].contiguous()
    buf, _ = sz.compress(f.cuda(), EB)
    want = sz.encode_cpu(f.numpy(), EB)
    assert (sz.to_container(buf, f.shape, EB).cpu().numpy() == want).all()


@pytest.mark.parametrize("value,eb", [(-50282496.0, 1.0), (-5028.2495, 1e-4)])   # 1.5 * 2^24 steps below 0: a tile of them has no codes
@pytest.mark.parametrize("nx", [256, 260, 257])
def test_tiles_that_begin_far_outside_the_codes_are_stored_raw(value, eb, nx):
    f = torch.randn((16, 24, nx), generator=torch.Generator().manual_seed(3)).cumsum(2) * (20 * eb)
    f[:8, 8:16, 32:64] = value
    f[8:, :8, 64:96] += value   # not constant, within 4094 codes of the first
    f[8:, 16:, 0] = value
    f[0, 0, 128] = value        # the first value alone
    f[1, 16, 200] = value       # another alone
    buf, _ = sz.compress(f.cuda(), eb)
    assert (sz.to_container(buf, f.shape, eb).cpu().numpy() == sz.encode_cpu(f.numpy(), eb)).all()
    assert (sz.decompress(buf, f.shape, eb).cpu() - f).abs().max() <= eb
