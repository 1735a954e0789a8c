"""The error-bounded codec where its accesses to a field change: lines on 32 bytes, on 16 and anywhere
(extents and a start of the buffer that allow no wider), tiles cut off in each direction, and packed
tiles from a few bytes to the largest that a warp stages (8256), against the host codec byte for byte."""
import numpy as np
import pytest
import torch

from ccbench_b200.ops import sz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 10, 40), (8, 8, 36), (17, 3, 33), (1, 1, 1), (3, 70, 31), (20, 16, 264)])
@pytest.mark.parametrize("start", [0, 4, 1])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 400.0, 1e5])   # widths of none, about 8, 16 and 24 bits at a bound of 1e-2
def test_bytes_and_values_at_every_line_width(shape, start, scale):
    n = int(np.prod(shape))
    host = torch.randn(n, generator=torch.Generator().manual_seed(n + start)) * scale
    field = torch.empty(n + start, device="cuda")[start:].copy_(host).view(shape)
    eb = 1e-2
    buf, used = sz.compress(field, eb)
    want = sz.encode_cpu(host.view(shape).numpy(), eb)
    assert np.array_equal(sz.to_container(buf, shape, eb).cpu().numpy(), want)
    assert int(used) == want.size - sz.HEADER_BYTES - 4 * (buf.numel() // sz.GROUP_STRIDE) - sz.GROUP_HEADER * (buf.numel() // sz.GROUP_STRIDE)
    out = torch.full((n + start + 8,), 7.0, device="cuda")
    target = out[start:start + n]
    sz._check(sz._decl().ccb_sz_decompress(buf.data_ptr(), shape[2], shape[1], shape[0], eb, target.data_ptr(), sz._stream()))
    torch.cuda.synchronize()
    assert np.array_equal(target.view(shape).cpu().numpy(), sz.decode_cpu(want))
    assert (out[:start] == 7).all() and (out[start + n:] == 7).all()


@pytest.mark.parametrize("damage", ["none", "short", "groups", "size", "payload", "magic"])
def test_container_opened_on_the_device(damage):
    shape, eb = (20, 30, 70), 1e-2
    field = torch.randn(shape, generator=torch.Generator().manual_seed(1)).cuda()
    buf, _ = sz.compress(field, eb)
    blob = sz.to_container(buf, shape, eb)
    words = blob[:sz.HEADER_BYTES + 8].view(torch.int32)
    if damage == "short":
        blob = blob[:sz.HEADER_BYTES + 60].clone()
    elif damage == "groups":      # more than the blob has room for
        words[7] = 1 << 30
    elif damage == "size":        # of the first group
        words[10] += 4
    elif damage == "payload":
        blob = blob[:-4].clone()
    elif damage == "magic":
        words[0] += 1
    if damage == "none":
        back, got_shape, got_eb = sz.from_container(blob)
        assert got_shape == shape and abs(got_eb - eb) < 1e-9
        assert torch.equal(sz.decompress(back, shape, got_eb), sz.decompress(buf, shape, eb))
        assert torch.equal(sz.to_container(back, shape, eb), blob)
    else:
        with pytest.raises(ValueError):
            sz.from_container(blob)


@pytest.mark.parametrize("start", [4, 8, 16])
def test_packed_and_raw_tiles_from_a_buffer_on_four_bytes(start):
    shape, eb = (17, 20, 96), 1e-2
    field = torch.randn(shape, generator=torch.Generator().manual_seed(2))
    field[:8, :8, 32:64] = 1e30
    buf, _ = sz.compress(field.cuda(), eb)
    moved = torch.empty(buf.numel() + start, dtype=torch.uint8, device="cuda")[start:]
    moved.copy_(buf)
    assert torch.equal(sz.decompress(moved, shape, eb), sz.decompress(buf, shape, eb))


@pytest.mark.parametrize("shape", [(17, 20, 96), (9, 9, 258), (9, 9, 32 * 1300), (9, 9, 32 * 1300 + 5)])   # a CTA a tile, a warp a tile
@pytest.mark.parametrize("word,value", [(0, 8 * 8256), (1, 12), (2, 1 << 31), (6, 7), (3, 0xfffffff0)])
def test_damaged_tile_sizes_stay_inside_the_slot(shape, word, value):
    """A size word that puts the tiles behind it where none can lie: those become NaN, the rest stay."""
    eb = 1e-2
    field = torch.randn(shape, generator=torch.Generator().manual_seed(3)).cuda()
    buf, _ = sz.compress(field, eb)
    want = sz.decompress(buf, shape, eb)
    bad = buf.clone()
    group = buf.numel() // sz.GROUP_STRIDE - 1
    sizes = bad[group * sz.GROUP_STRIDE:][:sz.GROUP_HEADER].view(torch.int32)
    sizes[word] = value if value < 1 << 31 else value - (1 << 32)
    words = [w & 0xffffffff for w in sizes.tolist()]
    got = sz.decompress(bad, shape, eb)
    with pytest.raises(ValueError):
        sz.to_container(bad, shape, eb)
    tx, ty = -(-shape[2] // 32), -(-shape[1] // 8)
    tiles = tx * ty * -(-shape[0] // 8)
    off = 0
    for t in range(tiles):
        z, y, x = 8 * (t // (tx * ty)), 8 * (t // tx % ty), 32 * (t % tx)
        box = (slice(z, z + 8), slice(y, y + 8), slice(x, x + 32))
        k = t % 8
        if t < 8 * group:
            continue
        if k <= word:
            assert torch.equal(got[box], want[box]), t
        elif off > k * sz.TILE_CAP or off % 16:
            assert got[box].isnan().all(), t
        got[box] = want[box]
        off = (off + words[k]) & 0xffffffff
    assert torch.equal(got, want)   # the groups before


@pytest.mark.parametrize("row", [0, 1, 31, 63])
@pytest.mark.parametrize("width", [33, 128, 254])
@pytest.mark.parametrize("nx", [64, 32 * 5200, 32 * 5200 - 3])
def test_damaged_row_widths_make_their_tile_nan(row, width, nx):
    shape, eb = (8, 8, nx), 1e-2
    field = torch.randn(shape, generator=torch.Generator().manual_seed(4)).cuda()
    buf, _ = sz.compress(field, eb)
    want = sz.decompress(buf, shape, eb)
    first = int(buf[:4].view(torch.int32))
    buf[sz.GROUP_HEADER + first + row] = width
    got = sz.decompress(buf, shape, eb)
    assert torch.equal(got[..., :32], want[..., :32]) and got[..., 32:64].isnan().all() and torch.equal(got[..., 64:], want[..., 64:])


@pytest.mark.parametrize("start", [0, 4])
@pytest.mark.parametrize("word,change", [(0, 4), (1, 16), (5, 1 << 20)])
def test_container_with_damaged_tile_sizes_is_refused_on_the_device(start, word, change):
    shape, eb = (20, 30, 70), 1e-2
    field = torch.randn(shape, generator=torch.Generator().manual_seed(1)).cuda()
    buf, _ = sz.compress(field, eb)
    blob = sz.to_container(buf, shape, eb)
    moved = torch.empty(blob.numel() + start, dtype=torch.uint8, device="cuda")[start:]
    moved.copy_(blob)
    assert torch.equal(sz.from_container(moved)[0], sz.from_container(blob)[0])
    first = int(blob[sz.HEADER_BYTES:][:4].view(torch.int32))
    at = sz.HEADER_BYTES + 4 * (buf.numel() // sz.GROUP_STRIDE) + first + 4 * word   # group 1
    moved[at:at + 4].view(torch.int32).add_(change)
    with pytest.raises(ValueError):
        sz.from_container(moved)


@pytest.mark.parametrize("nx", [64, 68, 65])
@pytest.mark.parametrize("z", [0, 1, 6, 7])
def test_tile_that_turns_out_raw_at_any_plane(nx, z):
    field = torch.randn(8, 8, nx, generator=torch.Generator().manual_seed(z)) * 1e4   # rows of about 22 bits before it
    field[z, 5, 37] = float("nan")
    buf, _ = sz.compress(field.cuda(), 1e-2)
    want = sz.encode_cpu(field.numpy(), 1e-2)
    assert np.array_equal(sz.to_container(buf, field.shape, 1e-2).cpu().numpy(), want)
    assert np.array_equal(sz.decompress(buf, field.shape, 1e-2).cpu().numpy(), sz.decode_cpu(want), equal_nan=True)


@pytest.mark.parametrize("ny", [8, 11])
@pytest.mark.parametrize("tail", [0, 8, 12, 31])   # lines on 32 bytes, on 16 and anywhere
@pytest.mark.parametrize("scale", [1e-3, 1.0, 400.0, 1e5])
@pytest.mark.parametrize("start", [0, 4])
def test_many_tiles_are_unpacked_as_few_are(ny, tail, scale, start):
    """A field that repeats a small one along x: more tiles than the kernel for few takes, each the tile
    of the small field (whose values are held against the host codec above). The last column is cut off."""
    nz, period, eb = 9, 64, 1e-2
    base = torch.randn((nz, ny, period), generator=torch.Generator().manual_seed(ny + tail)) * scale
    base[:8, :8, 32:] *= 1e-2
    base[8, 5, 40] = 1e30   # a raw tile
    repeats = 5200 // (2 * -(-nz // 8) * -(-ny // 8)) + 1
    field = torch.cat([base.repeat(1, 1, repeats), base[..., :tail]], -1).cuda()
    got_base = sz.decompress(sz.compress(base.cuda(), eb)[0], base.shape, eb)
    want = [got_base.repeat(1, 1, repeats)]
    if tail:
        want.append(sz.decompress(sz.compress(base[..., :tail].contiguous().cuda(), eb)[0], (nz, ny, tail), eb))
    buf, _ = sz.compress(field.contiguous(), eb)
    moved = torch.empty(buf.numel() + start, dtype=torch.uint8, device="cuda")[start:]
    moved.copy_(buf)
    assert torch.equal(sz.decompress(moved, field.shape, eb), torch.cat(want, -1))
